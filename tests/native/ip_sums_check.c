// The inner products' sums (shmoai_b200/csrc: AccDbl, Acc<true>) restated with IEEE double and 64-bit integer
// operations against 128-bit integers: random operands and operands at the ends of their ranges, every
// term count, primes at the edges.  Exit status 0 when all match.
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

typedef unsigned __int128 u128;
static uint64_t rng = 88172645463325252ull;
static uint64_t xs(void) { rng ^= rng << 13; rng ^= rng >> 7; rng ^= rng << 17; return rng; }
static const double magic = 6755399441055744.0, two52 = 4503599627370496.0, two103 = 10141204801825835211973625643008.0;
static uint64_t bits(double d) { uint64_t u; memcpy(&u, &d, 8); return u; }
static int range_bad;

static double centre(double v, double q, double qi) { return fma(-(fma(v, qi, magic) - magic), q, v); }
static double mul(double y, double w, double q, double qi) {
    const double hi = y * w, lo = fma(y, w, -hi), z = hi * qi;
    if (fabs(z) >= 2251799813685248.0) range_bad++;
    return fma(-(fma(hi, qi, magic) - magic), q, hi) + lo;
}

static uint64_t sum_dbl(const uint64_t *a, const uint64_t *b, int n, uint64_t Q) {
    const double q = (double)Q, qi = 1.0 / q;
    double H[2] = {1.5 * two103, 1.5 * two103}, L[2] = {0, 0};
    for (int i = 0; i < n; i++) {
        const double x = a[i] > Q / 2 ? (double)a[i] - q : (double)a[i], y = b[i] > Q / 2 ? (double)b[i] - q : (double)b[i];
        const double h = fma(x, y, H[i & 1]);
        if (h < two103 || h >= 2 * two103) range_bad++;
        L[i & 1] += fma(x, y, H[i & 1] - h);
        if (fabs(L[i & 1]) > 4503599627370496.0) range_bad++;
        H[i & 1] = h;
    }
    const double h = (H[0] - 1.5 * two103) + (H[1] - 1.5 * two103);
    const double c = centre(2251799813685248.0, q, qi) / 2251799813685248.0;
    const double t = mul(h, c, q, qi) + centre(L[0] + L[1], q, qi), r = centre(t, q, qi);
    return (uint64_t)(r < 0 ? r + q : r);
}

static uint64_t sum_52(const uint64_t *a, const uint64_t *b, int n, uint64_t Q) {
    const uint64_t m26 = (1u << 26) - 1;
    const double k = 67108864.0 * (1.0 / (double)Q);
    uint64_t lo = 0, mid = 0, hi = 0;
    for (int i = 0; i < n; i++) {
        const uint64_t a0 = a[i] & m26, a1 = a[i] >> 26, b0 = b[i] & m26, b1 = b[i] >> 26;
        lo += a0 * b0;
        mid += a0 * b1 + a1 * b0;
        hi += a1 * b1;
    }
    const double z1 = (double)hi * k;
    const uint64_t q1 = bits(fma((double)hi, k, two52)) & 0x000FFFFFFFFFFFFFull;
    const uint64_t m = (hi << 26) - q1 * Q + mid + (lo >> 26);
    const double z2 = (double)(int64_t)m * k;
    if (z1 >= 2251799813685248.0 || fabs(z2) >= 2251799813685248.0) range_bad++;
    const uint64_t q2 = bits(fma((double)(int64_t)m, k, magic)) - 0x4338000000000000ull;
    const uint64_t r = (m << 26) + (lo & m26) - q2 * Q;
    return r + ((uint64_t)((int64_t)r >> 63) & Q);
}

int main(void) {
    const uint64_t pd[] = {(1ull << 51) - 1, (1ull << 51) - (1ull << 13) + 1, (1ull << 50) + 1, (1ull << 46) - 1,
                           (1ull << 40) + 1, (1ull << 20) + 7};
    const uint64_t p5[] = {(1ull << 52) - 1, (1ull << 52) - (1ull << 17) + 1, (1ull << 51) + 1, (1ull << 46) - 1, (1ull << 40) + 1};
    int bad = 0;
    for (int kind = 0; kind < 2; kind++)
        for (int i = 0; i < (kind ? 5 : 6); i++) {
            const uint64_t Q = kind ? p5[i] : pd[i];
            int mis = 0;
            range_bad = 0;
            for (int it = 0; it < 40000; it++) {
                const int n = 1 + (int)(xs() % (kind ? 64 : 8)), mode = (int)(xs() % 4);
                uint64_t a[64], b[64], ref = 0;
                for (int t = 0; t < n; t++) {
                    const uint64_t e[4] = {0, Q / 2, Q / 2 + 1, Q - 1};
                    a[t] = mode & 1 ? e[xs() % 4] : xs() % Q;
                    b[t] = mode & 2 ? (mode == 3 && (it & 1) ? a[t] : e[xs() % 4]) : xs() % Q;
                    ref = (uint64_t)((ref + (u128)a[t] * b[t]) % Q);
                }
                mis += (kind ? sum_52 : sum_dbl)(a, b, n, Q) != ref;
            }
            printf("%s q=%llu: mismatches %d, out of range %d\n", kind ? "halves " : "doubles", (unsigned long long)Q, mis, range_bad);
            bad += mis + range_bad;
        }
    printf(bad ? "FAIL\n" : "OK\n");
    return bad != 0;
}

// The sums of products of shmoai_b200/csrc/modarith.cuh (Acc) restated with 64-bit integer and IEEE double
// operations against 128-bit integers, over the ranges each is used for: kAccHalves on residues of one prime from
// 2^28 up, kAccSplit on residues of one prime and on words below 2^52 times residues of another, of any size.
// Random operands and operands at the ends of their ranges, every term count.  Exit status 0 when all match.
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

typedef unsigned __int128 u128;
static uint64_t rng = 88172645463325252ull;
static uint64_t xs(void) { rng ^= rng << 13; rng ^= rng >> 7; rng ^= rng << 17; return rng; }
static uint64_t bits(double d) { uint64_t u; memcpy(&u, &d, 8); return u; }
static int range_bad;

static uint64_t halves(const uint64_t *a, const uint64_t *b, int n, uint64_t Q) {
    const double magic = 6755399441055744.0, two52 = 4503599627370496.0, two51 = 2251799813685248.0;
    const uint64_t m26 = (1u << 26) - 1;
    const double k = 67108864.0 * (1.0 / (double)Q);
    uint64_t lo = 0, mid = 0, hi = 0;
    for (int i = 0; i < n; i++) {
        const uint64_t a0 = a[i] & m26, a1 = a[i] >> 26, b0 = b[i] & m26, b1 = b[i] >> 26;
        lo += a0 * b0;
        mid += a0 * b1 + a1 * b0;
        hi += a1 * b1;
    }
    const uint64_t q1 = bits(fma((double)hi, k, two52)) & 0x000FFFFFFFFFFFFFull;
    const uint64_t m = (hi << 26) - q1 * Q + mid + (lo >> 26);
    if ((double)hi * k >= two51 || fabs((double)(int64_t)m * k) >= two51) range_bad++;
    const uint64_t q2 = bits(fma((double)(int64_t)m, k, magic)) - 0x4338000000000000ull;
    const uint64_t r = (m << 26) + (lo & m26) - q2 * Q;
    return r + ((uint64_t)((int64_t)r >> 63) & Q);
}

static uint64_t split(const uint64_t *a, const uint64_t *b, int n, uint64_t Q) {
    uint64_t lo = 0, mid = 0, hi = 0;
    for (int i = 0; i < n; i++) {
        const uint32_t a0 = (uint32_t)a[i], a1 = (uint32_t)(a[i] >> 32), b0 = (uint32_t)b[i], b1 = (uint32_t)(b[i] >> 32);
        const uint64_t t = (uint64_t)a0 * b0;
        lo += (uint32_t)t;
        mid += (t >> 32) + (uint64_t)a0 * b1 + (uint64_t)a1 * b0;
        hi += (uint64_t)a1 * b1;
    }
    const uint64_t l = lo + (mid << 32), h = hi + (mid >> 32) + (l < lo);
    const int kb = 64 - __builtin_clzll(Q);  // Barrett: the sum must stay below 2^(63 + k)
    if (kb + 63 < 128 && ((((u128)h << 64) | l) >> (kb + 63))) range_bad++;
    return (uint64_t)(((((u128)h << 64) | l)) % Q);
}

int main(void) {
    const uint64_t top = 1ull << 52;
    const uint64_t one[] = {(1ull << 28) + 1, (1ull << 28) + 4097, (1ull << 30) - 1, (1ull << 36) + 5, (1ull << 40) - 1,
                            (1ull << 46) - 1, top - 1};
    const uint64_t any[] = {(1ull << 20) - 3, (1ull << 28) + 1, (1ull << 39) + 1, (1ull << 40) - 1, (1ull << 46) - 1, top - 1};
    const char *name[] = {"halves", "split, words", "split, one prime"};
    int bad = 0;
    for (int kind = 0; kind < 3; kind++) {
        const uint64_t *qs = kind == 0 ? one : any;
        const int nq = kind == 0 ? 7 : 6, same = kind != 1;
        for (int i = 0; i < nq; i++) {
            const uint64_t Q = qs[i], lim = same ? Q : top;
            int mis = 0;
            range_bad = 0;
            for (int it = 0; it < 40000; it++) {
                const int n = 1 + (int)(xs() % (same ? 64 : 16)), mode = (int)(xs() % 4);
                uint64_t a[64], b[64], ref = 0;
                for (int t = 0; t < n; t++) {
                    const uint64_t ea[4] = {0, lim / 2, lim - (lim >> 26), lim - 1}, eb[4] = {0, Q / 2, Q - (Q >> 26), Q - 1};
                    a[t] = mode & 1 ? ea[mode == 3 ? 3 : xs() % 4] : xs() % lim;
                    b[t] = mode & 2 ? eb[mode == 3 ? 3 : xs() % 4] : xs() % Q;
                    ref = (uint64_t)((ref + (u128)a[t] * b[t]) % Q);
                }
                mis += (kind == 0 ? halves : split)(a, b, n, Q) != ref;
            }
            printf("%s q=%llu: mismatches %d, out of range %d\n", name[kind], (unsigned long long)Q, mis, range_bad);
            bad += mis + range_bad;
        }
    }
    printf(bad ? "FAIL\n" : "OK\n");
    return bad != 0;
}

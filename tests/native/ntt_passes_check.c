// The FP64 passes of both NTT directions (shmoai_b200/csrc/ntt.cuh: mul_dbl, fwd_pass_dbl, inv_pass_dbl)
// restated with IEEE double operations (compiled without contraction) and run beside exact integer
// arithmetic: 16 stages in passes of four (and 12 in passes of three), random twiddles and twiddles at
// +-(q-1)/2, random inputs and inputs at 0, q/2 and q-1.  Counts quotients outside the range in which
// the rounding through 1.5 2^52 is exact and values at or above 2^53.  Exit status 0 when all match.
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

typedef unsigned __int128 u128;
#define MAXN (1 << 16)
static uint64_t rng = 88172645463325252ull;
static uint64_t xs(void) { rng ^= rng << 13; rng ^= rng >> 7; rng ^= rng << 17; return rng; }
static const double magic = 6755399441055744.0;
static double q, qinv, maxz, maxv, maxt;
static uint64_t Q;

static void see(double v) { if (fabs(v) > maxv) maxv = fabs(v); }
static double mul(double y, double w) {
    const double hi = y * w, lo = fma(y, w, -hi);
    if (fabs(hi * qinv) > maxz) maxz = fabs(hi * qinv);
    const double k = fma(hi, qinv, magic) - magic;
    const double t = fma(-k, q, hi) + lo;
    if (fabs(t) > maxt) maxt = fabs(t);
    return t;
}
static double centre(double v) { return fma(-(fma(v, qinv, magic) - magic), q, v); }
static uint64_t canon(double v) { return (uint64_t)(v < 0 ? v + q : v); }

static uint64_t a[MAXN], w[MAXN];
static double d[MAXN], wd[MAXN];

// stage s of the forward transform: pairs N >> (s + 1) apart, twiddle (1 << s) + group
static int forward(int logn, int R, int centred) {
    const int n = 1 << logn;
    for (int i = 0; i < n; i++) {
        d[i] = (double)a[i];
        if (centred && a[i] > Q / 2) d[i] -= q;
    }
    for (int s = 0; s < logn; s++) {
        const int t = n >> (s + 1), last = s % R == R - 1;
        for (int i = 0; i < 1 << s; i++)
            for (int j = 2 * i * t; j < 2 * i * t + t; j++) {
                const uint64_t x = a[j], y = (uint64_t)((u128)a[j + t] * w[(1 << s) + i] % Q);
                a[j] = (x + y) % Q;
                a[j + t] = (x + Q - y) % Q;
                if (centred && last) d[j + t] = centre(d[j + t]);
                const double u = d[j], v = mul(d[j + t], wd[(1 << s) + i]);
                see(d[j] = u + v);
                see(d[j + t] = u - v);
            }
        if (centred && last && s < logn - 1)
            for (int k = 0; k < n; k++) d[k] = centre(d[k]);
    }
    int bad = 0;
    for (int k = 0; k < n; k++) bad += canon(centre(d[k])) != a[k];
    return bad;
}

// the inverse: stages logn-1 .. 0 in passes of R (the last one folded with a scale c, as the kernel does)
static int inverse(int logn, int R, int centred) {
    const int n = 1 << logn;
    static char small[MAXN];
    for (int i = 0; i < n; i++) { d[i] = (double)a[i]; small[i] = 0; }
    for (int s = logn - 1; s >= 0; s--) {
        const int t = n >> (s + 1), first = s % R == R - 1, end = s % R == 0;
        if (first) for (int k = 0; k < n; k++) small[k] = 0;  // a pass starts: nothing known
        for (int i = 0; i < 1 << s; i++)
            for (int j = 2 * i * t; j < 2 * i * t + t; j++) {
                const uint64_t x = a[j], y = a[j + t];
                const double u = d[j], v = d[j + t];
                if (s == 0) {  // scale c = w[0]: (x + y) c, (x - y) w c
                    const uint64_t c1 = (uint64_t)((u128)w[0] * w[1] % Q);
                    a[j] = (uint64_t)((u128)((x + y) % Q) * w[0] % Q);
                    a[j + t] = (uint64_t)((u128)((x + Q - y) % Q) * c1 % Q);
                    d[j] = mul(u + v, wd[0]);
                    d[j + t] = mul(u - v, c1 > Q / 2 ? (double)c1 - q : (double)c1);
                    continue;
                }
                a[j] = (x + y) % Q;
                a[j + t] = (uint64_t)((u128)((x + Q - y) % Q) * w[(1 << s) + i] % Q);
                see(u + v);
                see(u - v);
                d[j] = u + v;
                d[j + t] = mul(u - v, wd[(1 << s) + i]);
                if (centred) {
                    if (!small[j]) d[j] = centre(d[j]);
                    small[j] = !small[j];
                    small[j + t] = 0;
                }
            }
        // a pass's register index m = bits s+R-1 .. s of the element's position read from the top:
        // the values of index m < E / 4 are centred
        if (!centred && end && s > 0)
            for (int k = 0; k < n; k++)
                if (((k >> (logn - s - R)) & ((1 << R) - 1)) < (1 << R) / 4) d[k] = centre(d[k]);
    }
    int bad = 0;
    for (int k = 0; k < n; k++) bad += fabs(d[k]) >= q || canon(d[k]) != a[k];
    return bad;
}

static int run(uint64_t prime, int logn, int R) {
    Q = prime; q = (double)Q; qinv = 1.0 / q;
    const int centred = Q >= (1ull << 52) / 36, n = 1 << logn;
    int bad = 0;
    for (int kind = 0; kind < 4; kind++)
        for (int dir = 0; dir < 2; dir++) {
            maxz = maxv = maxt = 0;
            for (int i = 0; i < n; i++) {
                const uint64_t e[3] = {0, Q / 2, Q - 1};
                a[i] = kind & 1 ? e[xs() % 3] : xs() % Q;
                w[i] = kind & 2 ? (xs() & 1 ? Q / 2 : Q / 2 + 1) : xs() % Q;
                wd[i] = w[i] > Q / 2 ? (double)w[i] - q : (double)w[i];
            }
            const int m = dir ? inverse(logn, R, centred) : forward(logn, R, centred);
            const int range = maxz >= 2251799813685248.0 || maxv >= 9007199254740992.0;
            bad += m + range;
            printf("q=2^%.4f n=2^%d R=%d kind %d %s: mismatches %d, out of range %d (|z| 2^%.2f, |v| %.2f q, |t| %.3f q)\n",
                   log2(q), logn, R, kind, dir ? "inverse" : "forward", m, range, log2(maxz), maxv / q, maxt / q);
        }
    return bad;
}

int main(void) {
    const uint64_t lim = (1ull << 52) / 36;
    const uint64_t p[] = {lim - 1 - lim % 2, (1ull << 46) - (1ull << 17) + 1, (1ull << 30) + 1, lim + 1 + lim % 2,
                          (1ull << 50) + (1ull << 17) + 1, (1ull << 51) - (1ull << 17) + 1};
    int bad = 0;
    for (int i = 0; i < 6; i++) bad += run(p[i] | 1, 16, 4) + run(p[i] | 1, 12, 3);
    printf(bad ? "FAIL\n" : "OK\n");
    return bad != 0;
}

// Batched negacyclic NTT / INTT over RNS limbs.
//
// Definition (bit-identical to the reference, thirdparty/phantom-fhe/src/ntt/fntt_2d.cu
// and intt_2d.cu): forward = Cooley-Tukey with root_powers[bitrev(i)] = psi^i, natural
// order in, bit-reversed order out, fully reduced to [0, q); inverse = Gentleman-Sande
// with psi^-i, including N^-1.
//
// Decomposition: N = M * M (M = 2^(2R)).  The first log M forward stages only
// combine elements of one "column" {c + M*p : p < M}; the last log M stages only
// combine elements of one contiguous "block" {b*M + p : p < M}.  Each phase is one
// kernel in which a CTA owns S columns (or S blocks) of one limb (S = 16 or 8, the tile
// variant); a thread owns 2^R elements and runs R radix-2 stages in registers, twice, with
// one shared-memory exchange in between.  Global loads and stores move S consecutive words
// per column row / per block segment (128 bytes at S = 16).  Values between the two
// phases are lazy: below 36q (grow butterflies, q < 2^57), in [0, 4q) (Harvey), or signed
// doubles (the FP64 butterflies, q < 2^51).
//
// The inverse's last stage folds a per-limb scale c (N^-1, or N^-1 times the
// ModUp digit factor) into both outputs: (X+Y)*c and (X-Y)*psi^-(N/2)*c.
#pragma once
#include <cstdint>

#include "modarith.cuh"

namespace shm {

// Tile variants of the NTT kernels (columns or blocks per CTA, minimum resident CTAs per SM,
// which caps the registers a thread may use); the autotuner picks one per context.
struct NttVariant {
    int subs, min_blocks;
};
constexpr NttVariant kNttVariants[] = {{16, 4}, {16, 3}, {8, 8}, {8, 6}};
constexpr int kNttVariantCount = 4;
// The tile until one is tuned or set: 8 x 6 (80 registers, no spills; the small tile spreads few rows more
// evenly).  Its share of the time at 16 x 4, medians of alternated runs: forward and inverse of 117 x 35 limbs
// 0.91, a product at 24 limbs 0.92 (333 of 362 us), five rotations at 17 limbs 0.96, sixteen products at 27 limbs
// 0.98; 8 x 5 and 8 x 7 lie between.
constexpr int kNttDefault = 3;

// The rows a launch transforms: slots [first, first + count) of each of `polys` polynomials of
// `slots` limbs.  Slot s stands at position j = s % lp of its digit s / lp (lp = slots: one digit)
// and uses prime j below lq, else the special prime nq + j - lq.  skip > 0 (ModUp): the limbs
// [d skip, min((d + 1) skip, lq)) of digit d are left alone.
struct NttRows {
    uint32_t polys = 0, slots = 0, first = 0, count = 0, lp = 0, lq = 0, nq = 0, skip = 0;
};
constexpr uint32_t kNoPrime = 0xffffffffu;

__host__ __device__ __forceinline__ uint32_t row_prime(const NttRows &r, uint32_t slot) {
    const uint32_t j = slot % r.lp;
    if (r.skip) {
        const uint32_t s0 = slot / r.lp * r.skip;
        if (j >= s0 && j < s0 + r.skip && j < r.lq) return kNoPrime;
    }
    return j < r.lq ? j : r.nq + (j - r.lq);
}

// The rescale's forward NTT (ntt_forward_rescale): rows (poly, j < L-1) are read as
// last[poly] mod q_j and written as (in[poly][j] - NTT(...)) * q_{L-1}^-1 into out[poly][j]
struct RescaleIO {
    const uint64_t *last = nullptr;  // [polys][N], c_{L-1} in coefficient form
    const uint64_t *in = nullptr;    // [polys][L][N]
    uint64_t *out = nullptr;         // [polys][L-1][N]
    const uint64_t *inv = nullptr;   // [L-1][2]: q_{L-1}^-1 mod q_j and its Shoup companion
};

// The ModDown's forward NTT (ntt_forward_moddown): rows (poly, j < L) of the delta buffer are the base
// conversion sum_k z_k (phat_k mod q_j) of the INTT'd special-prime limbs z_k = acc[poly][L + k] (left there by
// conv_rows when `bytes` is given, else formed by the column phase's loads), and written as
// (acc[poly][j] - NTT(...)) P^-1 (+ add, or + add * add_mul[j]) into out;
// poly = ct * H + h.  The add term of rows h < n_add is read at perm[pos] for rows h < n_perm.
struct ModDownIO {
    const uint64_t *acc = nullptr;   // [polys][L + np][N]
    const uint64_t *conv = nullptr;  // [nq][np]: phat_k mod q_j
    const uint64_t *pinv = nullptr;  // [nq][2]: P^-1 mod q_j and its Shoup companion
    uint64_t *out = nullptr;
    const uint64_t *add = nullptr;
    const uint64_t *add_mul = nullptr;  // [nq][2]: the add term times this per-limb constant; null: as is
    const uint32_t *perm = nullptr;
    // exact conversion: the conversion sum minus vs[j][v] (v S mod q_j) with v = vrow[poly][k],
    // the overflow count floor(sum_k z_k / s_k); null: the approximate conversion
    const uint8_t *vrow = nullptr;
    const uint64_t *vs = nullptr;  // [slots][16]
    long long out_ct = 0, out_h = 0, add_ct = 0, add_h = 0;  // word strides
    uint32_t H = 2, np = 0, n_add = 0, n_perm = 0;
    int sums = 0;  // Context::split_acc
    const uint8_t *bytes = nullptr;  // the conversion's (and v's) constants for ConvIO; null: the load transform
};

// ModUp's forward NTT (ntt_forward_modup): row (ct, b, j) of up [n_cts][beta][LP][N].  For j
// outside digit b (limbs [b alpha, min((b+1) alpha, L))) the row is the base conversion
// sum_i y_i (qhat_i mod t_j) of the digit's INTT'd, qhat^-1-scaled limbs y = x[ct][b alpha ..] (coefficient form;
// left in up by conv_rows when `bytes` is given, else formed by the column phase's loads) and is transformed;
// rows j inside the digit are left alone (NttRows::skip).
struct ModUpIO {
    const uint64_t *x = nullptr;     // [n_cts][L][N]
    const uint64_t *conv = nullptr;  // [beta][LP][np]: qhat_i mod t_j of the level's digits
    uint32_t L = 0, np = 0, LP = 0;
    int sums = 0;
    const uint8_t *bytes = nullptr;  // as ModDownIO's
};

// The same conversions with the products on the tensor cores (conv.cu).  Set s (ciphertext
// s / per, digit s % per) has the coefficient-form limbs y_i at src + ct src_ct + (digit na + i) N,
// i < na (fewer in the last digit: total limbs in all); output row j (prime j below lq, else
// nq + j - lq) is sum_i y_i c_ij, plus v c_(na)j when an overflow count v is given per coefficient,
// at out[s][j] in the form the row's butterflies take; with skip_own a row j of the digit's own limbs is left alone.
// bytes: [per][rows][512], row j's constants: byte o of (c_ij 2^(8b) mod q_j) at
// (k / 16) 128 + 16 o + k % 16, k = 8 i + b.
constexpr uint32_t kConvSlots = 8;  // limbs and overflow count of a set
struct ConvIO {
    const uint64_t *src = nullptr;
    size_t src_ct = 0;
    const uint8_t *bytes = nullptr;
    uint64_t *out = nullptr;
    const uint8_t *vrow = nullptr;  // [sets][N]
    uint32_t sets = 0, per = 1, na = 1, total = 1, rows = 0, lq = 0, nq = 0;
    bool skip_own = false;
    __host__ __device__ __forceinline__ uint32_t prime(uint32_t j) const { return j < lq ? j : nq + (j - lq); }
};

// the optional load / store transforms of the forward NTT kernels
struct NttIO {
    RescaleIO rs;
    ModDownIO md;
    ModUpIO mu;
    int converted = 0;  // ModUp, ModDown: the rows have been converted (conv_rows)
};
constexpr int kIoPlain = 0, kIoRescale = 1, kIoModDown = 2, kIoModUp = 3, kIoConverted = 4;

__device__ __forceinline__ void ct_bf(uint64_t &x, uint64_t &y, uint64_t w, uint64_t ws, uint64_t q) {
    uint64_t q2 = 2 * q;
    uint64_t a = csub(x, q2);
    uint64_t t = shoup_lazy(y, w, ws, q);
    x = a + t;
    y = a - t + q2;
}

// Cooley-Tukey butterfly without the reduction of x: outputs exceed the inputs by less
// than 4q (shoup_lazy4 is below 4q for any 64-bit multiplicand).  From inputs below 4q,
// 16 stages stay below 68q < 2^(k+7), so this is exact for primes q < 2^57 and the last
// stage's output is reduced by reduce_small.
constexpr uint64_t kGrowPrimeLimit = 1ull << 57;

__device__ __forceinline__ void ct_bf_grow(uint64_t &x, uint64_t &y, uint64_t w, uint64_t ws, uint64_t q) {
    uint64_t t = shoup_lazy4(y, w, ws, q);
    uint64_t a = x;
    x = a + t;
    y = a - t + 4 * q;
}

// ---- FP64 butterflies (primes below 2^51)
//
// Both directions of the transform run on the FP64 pipe for primes below kF64CentreLimit, on values
// held as doubles (signed exact integers, in the uint64_t registers as their bit patterns; the first
// phase's output keeps that form in memory for the second).  The product of y with a twiddle w, kept
// within q/2 of zero, is t = y w - Q q with Q = round(hi / q): hi = y w rounded, lo = y w - hi exactly
// (an fma), Q from fma(hi, qinv, 1.5 2^52), hi - Q q exact by another fma (an integer below 2^53), and
// t = (hi - Q q) + lo exact: six FP64 operations, no integer multiply and one table word per twiddle.
// With z = y w / q, |Q - z| <= 1/2 + |z| 2^-52 (the roundings of hi and of qinv = 1 / q), so
// |t| <= q (1/2 + |y| 2^-53), for |z| < 2^51 (the rounding through 1.5 2^52 is then exact).
//
// What bounds it: the FP64 pipe (eight operations per butterfly and, for 51-bit primes, three per
// centring) and HBM (each phase reads and writes every limb) within 1.5x of each other.  117 x 35
// limbs at the bootstrapping primes, forward of one batch and inverse of another, 16 x 4 tiles: 5.56 ms
// with two table words per forward twiddle and integer Gentleman-Sande butterflies (whose low products
// kept the integer-multiply pipe busy), 4.06 ms so (3.80 at 8 x 6).
//
// kBfF64, q < 2^52 / 36.  Forward: inputs below q, a stage adds less than 0.65 q, values stay below
// 11 q over all 16 stages with no reduction.  Inverse (x + y, (x - y) w): from inputs below 1.8 q a
// pass of four stages grows the value at index 0 to at most 29 q < 2^52, the product of any
// difference stays below 0.9 q; indices 0 .. 3 (0 and 1 of a three-stage pass), which were last
// multiplied two or more stages before the pass's end, are centred at its end, the others stay
// below 1.8 q.
//
// kBfF64R, q < 2^51 (values below 4 q are exact).  Forward: values within q/2 of zero at the start of
// a pass, three stages leave them below 1.13 q, 1.91 q and 2.88 q; the multiplicands of the pass's
// last stage are centred before their products (a multiplicand must stay below 2 q), its outputs
// stay below 3.51 q, and every value is centred for the next pass.  Inverse: values stay below
// q + 3 at every stage: a sum of two such values is centred, a sum of two centred values is not.
constexpr uint64_t kF64GrowLimit = (1ull << 52) / 36;
constexpr uint64_t kF64CentreLimit = 1ull << 51;
constexpr double kTwo52 = 4503599627370496.0, kMagic = 6755399441055744.0;  // 2^52, 1.5 2^52

__device__ __forceinline__ double as_dbl(uint64_t x) { return __longlong_as_double((long long)x); }
__device__ __forceinline__ uint64_t as_bits(double x) { return (uint64_t)__double_as_longlong(x); }

// y w mod q as a signed value (see above)
__device__ __forceinline__ double mul_dbl(double y, double w, double q, double qinv) {
    const double hi = __dmul_rn(y, w);
    const double lo = __fma_rn(y, w, -hi);
    const double Q = __dsub_rn(__fma_rn(hi, qinv, kMagic), kMagic);
    return __dadd_rn(__fma_rn(-Q, q, hi), lo);
}

__device__ __forceinline__ void ct_bf_dbl(uint64_t &xb, uint64_t &yb, double w, double q, double qinv) {
    const double x = as_dbl(xb), t = mul_dbl(as_dbl(yb), w, q, qinv);
    xb = as_bits(__dadd_rn(x, t));
    yb = as_bits(__dsub_rn(x, t));
}

__device__ __forceinline__ void gs_bf_dbl(uint64_t &xb, uint64_t &yb, double w, double q, double qinv) {
    const double x = as_dbl(xb), y = as_dbl(yb);
    xb = as_bits(__dadd_rn(x, y));
    yb = as_bits(mul_dbl(__dsub_rn(x, y), w, q, qinv));
}

// x < 2^52 as the double x
__device__ __forceinline__ double to_dbl(uint64_t x) { return __dsub_rn(as_dbl(0x4330000000000000ull | x), kTwo52); }

// x in [0, q) as a double within q/2 of zero
__device__ __forceinline__ double to_dbl_centred(uint64_t x, uint64_t q) {
    return __dsub_rn(as_dbl(0x4330000000000000ull | x), x > (q >> 1) ? __dadd_rn(kTwo52, (double)q) : kTwo52);
}

// v (|v| < 2^53, a signed integer) -> v - round(v / q) q, within q/2 + 1 of zero, exact
__device__ __forceinline__ double dbl_centre(double v, double q, double qinv) {
    const double Q = __dsub_rn(__fma_rn(v, qinv, kMagic), kMagic);
    return __fma_rn(-Q, q, v);
}

// |v| < q -> v mod q in [0, q) as an integer (2^52 + q is exact: q < 2^51)
__device__ __forceinline__ uint64_t dbl_canon(double v, double q) {
    const double r = __dadd_rn(v, (int)(as_bits(v) >> 32) < 0 ? __dadd_rn(kTwo52, q) : kTwo52);
    return as_bits(r) & 0x000FFFFFFFFFFFFFull;
}

// a signed integer |v| < 2^53 -> v mod q in [0, q)
__device__ __forceinline__ uint64_t dbl_mod(double v, double q, double qinv) {
    return dbl_canon(dbl_centre(v, q, qinv), q);
}

// Sum of up to eight products of centred residues (to_dbl_centred) of a prime below 2^51, on the FP64 pipe.
// H starts at 1.5 2^103, where doubles are multiples of 2^51: H' = H + a b rounded, the step H' - H is exact,
// and so is the rest a b - (H' - H) (an integer, at most 2^50), which goes to L.  Two chains of four
// products (each below 2^100) keep H inside [2^103, 2^104) and L below 2^53 in all.  At the end
// h = H - 1.5 2^103 (both chains: 2^51 times an integer below 2^52) is taken mod q as a product with
// 2^51 mod q and L is centred.  Four operations a term on a pipe that takes 64 a clock per SM; as 32-bit
// halves a term is four wide multiply-adds at 32 a clock.
constexpr int kMaxDblTerms = 8;
constexpr double kTwo103 = 10141204801825835211973625643008.0;  // 2^103
struct AccDbl {
    double H[2] = {1.5 * kTwo103, 1.5 * kTwo103}, L[2] = {0.0, 0.0};
    __device__ __forceinline__ void add(int i, double a, double b) {  // term i
        const double h = __fma_rn(a, b, H[i & 1]);
        L[i & 1] = __dadd_rn(L[i & 1], __fma_rn(a, b, __dsub_rn(H[i & 1], h)));
        H[i & 1] = h;
    }
    // c = 2^51 mod q within q/2 + 1 of zero, times 2^-51
    __device__ __forceinline__ uint64_t reduce(double q, double qinv, double c) const {
        const double h = __dadd_rn(__dsub_rn(H[0], 1.5 * kTwo103), __dsub_rn(H[1], 1.5 * kTwo103));
        return dbl_mod(__dadd_rn(mul_dbl(h, c, q, qinv), dbl_centre(__dadd_rn(L[0], L[1]), q, qinv)), q, qinv);
    }
    __device__ __forceinline__ static double two51_mod(double q, double qinv) {
        return __dmul_rn(dbl_centre(2251799813685248.0, q, qinv), 1.0 / 2251799813685248.0);
    }
};

__device__ __forceinline__ void gs_bf(uint64_t &x, uint64_t &y, uint64_t w, uint64_t ws, uint64_t q) {
    uint64_t q2 = 2 * q;
    uint64_t a = x + y;
    uint64_t d = x - y + q2;
    x = csub(a, q2);
    y = shoup_lazy(d, w, ws, q);
}

// Gentleman-Sande butterfly on [0, 4q) with the cheaper quotient of shoup_lazy4 (needs 8q < 2^64)
__device__ __forceinline__ void gs_bf4(uint64_t &x, uint64_t &y, uint64_t w, uint64_t ws, uint64_t q) {
    uint64_t q4 = 4 * q;
    uint64_t a = x + y;
    uint64_t d = x - y + q4;
    x = csub(a, q4);
    y = shoup_lazy4(d, w, ws, q);
}

// The butterfly family of a limb's prime, both directions.  kBfHarvey: values in [0, 4q) forward,
// [0, 2q) inverse (any prime); kBfGrow: ct_bf_grow / gs_bf4 (below kGrowPrimeLimit).
constexpr int kBfHarvey = 0, kBfGrow = 1, kBfF64 = 2, kBfF64R = 3;

__host__ __device__ __forceinline__ int bf_mode_of(uint64_t q) {
    return q < kF64GrowLimit ? kBfF64 : q < kF64CentreLimit ? kBfF64R : q < kGrowPrimeLimit ? kBfGrow : kBfHarvey;
}

// The families a kernel instantiation carries (a bit per family).  Every unrolled family adds a full
// copy of the transform's butterflies to the kernel, so a context's launches use the instantiation
// with just the families its primes need: kFamSmall (every prime below 2^51: the bootstrapping
// chains), kFamLarge (none below kF64GrowLimit), kFamAll otherwise.
constexpr int kFamSmall = (1 << kBfF64) | (1 << kBfF64R),
              kFamLarge = (1 << kBfF64R) | (1 << kBfGrow) | (1 << kBfHarvey), kFamAll = kFamSmall | kFamLarge;
__host__ __device__ constexpr bool fam_has(int fam, int mode) { return (fam >> mode) & 1; }
constexpr bool fam_fp(int fam) { return fam & kFamSmall; }
constexpr bool fam_int(int fam) { return fam & ((1 << kBfGrow) | (1 << kBfHarvey)); }

// ---- FP64 twiddle tables: per prime and direction N / 2^R + N doubles (N = 2^(4R)), within q/2 of zero.
// The first 2^(3R) entries are the bit-reversed table's (the column phase and the block phase's
// first pass, whose threads read one entry per block or per column).  The rest are the block
// phase's second pass, whose threads each need 2^R - 1 entries of their own: stage r of block b,
// thread g reads entries ((M + b) 2^R + g) 2^r + i, i < 2^r, which lie 2^r words apart for
// neighbouring threads.  They are stored as slots 2^r + i of a row of 2^R (slot 0 unused), slots
// in pairs, pairs thread-minor: [b][slot / 2][g][slot % 2], so that a half-warp reads 256 contiguous
// bytes: 16-byte loads of neighbouring threads instead of 8-byte loads up to 64 bytes apart
// (the second pass's table loads were 340 of about 570 L1 wavefronts per warp of fwd_blk).
template <int R>
struct TwTab {
    static constexpr uint32_t E = 1u << R, M = 1u << (2 * R), N = 1u << (4 * R), NAT = 1u << (3 * R);
    static constexpr size_t DIR = (size_t)N + NAT;  // doubles per prime and direction
    __host__ __device__ static size_t slot(uint32_t b, uint32_t g, uint32_t s) {
        return NAT + (((size_t)b * (E / 2) + (s >> 1)) * E + g) * 2 + (s & 1);
    }
};

// entries (u << r) + i of the natural part
struct TwNatural {
    const double *p;
    uint32_t u;
    __device__ __forceinline__ double one() const { return __ldg(p + u); }
    __device__ __forceinline__ double2 pair(int r, int i) const {
        return __ldg(reinterpret_cast<const double2 *>(p + ((u << r) + i)));
    }
};

// the second block pass's slots of one thread (p = table of the prime and direction)
template <int R>
struct TwLane {
    const double2 *p;
    __device__ __forceinline__ TwLane(const double *t, uint32_t b, uint32_t g)
        : p(reinterpret_cast<const double2 *>(t + TwTab<R>::slot(b, g, 0))) {}
    __device__ __forceinline__ double one() const { return __ldg(reinterpret_cast<const double *>(p) + 1); }
    __device__ __forceinline__ double2 pair(int r, int i) const {
        return __ldg(p + (size_t)((((1 << r) + i) >> 1) << R));
    }
};

// R forward stages on E = 2^R registers; stage r's pair starting at m uses entry m >> (R - r) of the
// stage's 2^r.  LAST: the block phase's second pass, whose values are reduced by the caller.
template <int R, bool CENTRED, bool LAST, class TW>
__device__ __forceinline__ void fwd_pass_dbl(uint64_t (&a)[1 << R], const TW &tw, double q, double qinv) {
    constexpr int E = 1 << R;
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int half = E >> (r + 1);
#pragma unroll
        for (int i = 0; i < (1 << r); i += 2) {
            double2 w = r == 0 ? make_double2(tw.one(), 0.0) : tw.pair(r, i);
#pragma unroll
            for (int k = 0; k < (r == 0 ? 1 : 2); k++) {
#pragma unroll
                for (int h = 0; h < half; h++) {
                    const int m = (i + k) * 2 * half + h;
                    if (CENTRED && r == R - 1) a[m + half] = as_bits(dbl_centre(as_dbl(a[m + half]), q, qinv));
                    ct_bf_dbl(a[m], a[m + half], k ? w.y : w.x, q, qinv);
                }
            }
        }
    }
    if (CENTRED && !LAST) {
#pragma unroll
        for (int m = 0; m < E; m++) a[m] = as_bits(dbl_centre(as_dbl(a[m]), q, qinv));
    }
}

// R inverse stages; skip_stage0 leaves the last one (the transform's final stage) to the caller.
// Which values are centred is decided at compile time (see the bounds above).
template <int R, bool CENTRED, bool SKIP0, class TW>
__device__ __forceinline__ void inv_pass_dbl(uint64_t (&a)[1 << R], const TW &tw, double q, double qinv) {
    constexpr int E = 1 << R;
    bool small[E];  // within q/2 + 1 of zero
#pragma unroll
    for (int m = 0; m < E; m++) small[m] = false;
#pragma unroll
    for (int r = R - 1; r >= (SKIP0 ? 1 : 0); r--) {
        const int half = E >> (r + 1);
#pragma unroll
        for (int i = 0; i < (1 << r); i += 2) {
            double2 w = r == 0 ? make_double2(tw.one(), 0.0) : tw.pair(r, i);
#pragma unroll
            for (int k = 0; k < (r == 0 ? 1 : 2); k++) {
#pragma unroll
                for (int h = 0; h < half; h++) {
                    const int m = (i + k) * 2 * half + h;
                    gs_bf_dbl(a[m], a[m + half], k ? w.y : w.x, q, qinv);
                    if (CENTRED) {
                        const bool c = !small[m];
                        if (c) a[m] = as_bits(dbl_centre(as_dbl(a[m]), q, qinv));
                        small[m] = c;
                        small[m + half] = false;
                    }
                }
            }
        }
    }
    if (!CENTRED && !SKIP0) {
#pragma unroll
        for (int m = 0; m < E / 4; m++) a[m] = as_bits(dbl_centre(as_dbl(a[m]), q, qinv));
    }
}

// the integer families: stage r of the pass is global stage s0 + r, the twiddle of the pair starting
// at m is entry (u << r) + (m >> (R - r)), u = (tb << s0) + g
template <int R, int MODE>
__device__ __forceinline__ void fwd_pass_int(uint64_t (&a)[1 << R], const uint64_t *__restrict__ w,
                                             const uint64_t *__restrict__ ws, uint32_t u, uint64_t q) {
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int half = (1 << R) >> (r + 1);
#pragma unroll
        for (int m = 0; m < (1 << R); m++) {
            if (m & half) continue;
            const uint32_t idx = (u << r) + (m >> (R - r));
            if (MODE == kBfGrow)
                ct_bf_grow(a[m], a[m + half], __ldg(w + idx), __ldg(ws + idx), q);
            else
                ct_bf(a[m], a[m + half], __ldg(w + idx), __ldg(ws + idx), q);
        }
    }
}

template <int R, int MODE, bool SKIP0>
__device__ __forceinline__ void inv_pass_int(uint64_t (&a)[1 << R], const uint64_t *__restrict__ w,
                                             const uint64_t *__restrict__ ws, uint32_t u, uint64_t q) {
#pragma unroll
    for (int r = R - 1; r >= (SKIP0 ? 1 : 0); r--) {
        const int half = (1 << R) >> (r + 1);
#pragma unroll
        for (int m = 0; m < (1 << R); m++) {
            if (m & half) continue;
            const uint32_t idx = (u << r) + (m >> (R - r));
            if (MODE == kBfGrow)
                gs_bf4(a[m], a[m + half], __ldg(w + idx), __ldg(ws + idx), q);
            else
                gs_bf(a[m], a[m + half], __ldg(w + idx), __ldg(ws + idx), q);
        }
    }
}

// a pass in the family `mode` (uniform per CTA: one limb), one of the families FAM carries
template <int R, int FAM, bool LAST, class TW>
__device__ __forceinline__ void fwd_pass(int mode, uint64_t (&a)[1 << R], const TW &tw, double qd, double qinv,
                                         const uint64_t *__restrict__ w, const uint64_t *__restrict__ ws, uint32_t u,
                                         uint64_t q) {
    if (fam_has(FAM, kBfF64) && mode == kBfF64)
        fwd_pass_dbl<R, false, LAST>(a, tw, qd, qinv);
    else if (fam_has(FAM, kBfF64R) && (FAM == kFamSmall || mode == kBfF64R))
        fwd_pass_dbl<R, true, LAST>(a, tw, qd, qinv);
    else if (fam_has(FAM, kBfGrow) && mode == kBfGrow)
        fwd_pass_int<R, kBfGrow>(a, w, ws, u, q);
    else if (fam_has(FAM, kBfHarvey))
        fwd_pass_int<R, kBfHarvey>(a, w, ws, u, q);
}

template <int R, int FAM, bool SKIP0, class TW>
__device__ __forceinline__ void inv_pass(int mode, uint64_t (&a)[1 << R], const TW &tw, double qd, double qinv,
                                         const uint64_t *__restrict__ w, const uint64_t *__restrict__ ws, uint32_t u,
                                         uint64_t q) {
    if (fam_has(FAM, kBfF64) && mode == kBfF64)
        inv_pass_dbl<R, false, SKIP0>(a, tw, qd, qinv);
    else if (fam_has(FAM, kBfF64R) && (FAM == kFamSmall || mode == kBfF64R))
        inv_pass_dbl<R, true, SKIP0>(a, tw, qd, qinv);
    else if (fam_has(FAM, kBfGrow) && mode == kBfGrow)
        inv_pass_int<R, kBfGrow, SKIP0>(a, w, ws, u, q);
    else if (fam_has(FAM, kBfHarvey))
        inv_pass_int<R, kBfHarvey, SKIP0>(a, w, ws, u, q);
}

}  // namespace shm

// The NTT kernels (see ntt.cuh for the decomposition) and their launches, a template over the ring
// (R: N = 2^(4R)) and the butterfly families; every instantiation is a translation unit of its own.
#pragma once
#include <algorithm>

#include "core.hpp"

namespace shm {

template <int R, int S>
struct Geo {
    static constexpr int LOGM = 2 * R;
    static constexpr uint32_t M = 1u << LOGM;  // sub-transform length
    static constexpr int LOGN = 2 * LOGM;
    static constexpr uint32_t N = 1u << LOGN;
    static constexpr int E = 1 << R;  // elements per thread
    static constexpr uint32_t THREADS = S * E;
    static constexpr uint32_t CHUNKS = M / S;  // CTAs per limb
    static constexpr uint32_t PAD_M = M + M / 16;     // padded block row in shared memory
};

__device__ __forceinline__ uint32_t padded(uint32_t p) { return p + (p >> 4); }

// what a CTA knows of its limb: tables of the prime and its constants
template <int R>
struct Limb {
    uint64_t q;
    double qd, qinv;
    int mode;
    const uint64_t *w, *ws;  // integer families: the twiddles and their Shoup companions
    const double *t;         // FP64 families: TwTab
    __device__ __forceinline__ Limb(uint32_t pidx, bool inverse, const uint64_t *tw, const double *twd,
                                    const PrimeConst *pc) {
        const PrimeConst &p = pc[pidx];
        q = p.q;
        qd = (double)q;
        qinv = p.qinv;
        mode = bf_mode_of(q);
        w = tw + ((size_t)pidx * 4 + (inverse ? 2 : 0)) * TwTab<R>::N;
        ws = w + TwTab<R>::N;
        t = twd + ((size_t)pidx * 2 + (inverse ? 1 : 0)) * TwTab<R>::DIR;
    }
    __device__ __forceinline__ bool fp() const { return mode == kBfF64 || mode == kBfF64R; }
};

// sum_{i < n} x[i << log_n] c[i] mod p (a base conversion's term for one coefficient; n <= 16).  The
// first eight terms' loads are issued together before any product, so one load latency is exposed
// per coefficient instead of one per term.
template <int KIND>
__device__ __forceinline__ uint64_t conv_sum(const uint64_t *__restrict__ x, const uint64_t *c, uint32_t n,
                                             int log_n, const PrimeConst &p) {
    constexpr uint32_t kBatch = 8;
    uint64_t v[kBatch];
#pragma unroll
    for (uint32_t i = 0; i < kBatch; i++) v[i] = i < n ? x[(size_t)i << log_n] : 0;
    Acc<KIND> acc;
#pragma unroll
    for (uint32_t i = 0; i < kBatch; i++)
        if (i < n) acc.add(v[i], c[i]);
    for (uint32_t i = kBatch; i < n; i++) acc.add(x[(size_t)i << log_n], c[i]);
    return acc.reduce(p);
}

__device__ __forceinline__ uint64_t conv_sum(int kind, const uint64_t *__restrict__ x, const uint64_t *c, uint32_t n,
                                             int log_n, const PrimeConst &p) {
    return kind == kAccSplit ? conv_sum<kAccSplit>(x, c, n, log_n, p) : conv_sum<kAccWide>(x, c, n, log_n, p);
}

// CTAs are issued limb-major: consecutive CTAs work on the same slot (one prime) of successive
// polynomials, so the CTAs in flight share one prime's twiddle table in L2.  CTA row t -> polynomial
// t % polys, slot first + t / polys.

// ---------------- forward, phase 1: columns (global stages 0 .. LOGM-1)
// IOK = kIoRescale: row (poly, j) is read as c_last[poly] mod q_j from the coefficient-form
// last limbs; kIoModDown: as the base conversion of the special-prime limbs (ModDownIO);
// kIoPlain: from `data`; kIoConverted: from `data`, as conv_rows leaves it
template <int R, int S, int MINB, int IOK, int FAM>
__global__ void __launch_bounds__(Geo<R, S>::THREADS, MINB)
    fwd_col(uint64_t *__restrict__ data, NttRows rw, const uint64_t *__restrict__ tw, const double *__restrict__ twd,
            const PrimeConst *__restrict__ pc, NttIO io) {
    using G = Geo<R, S>;
    __shared__ uint64_t sm[G::M * S];
    const uint32_t chunk = blockIdx.x % G::CHUNKS, t = blockIdx.x / G::CHUNKS;
    // ModUp rows go ct-major instead: the rows of one digit are consecutive CTAs, so the digit's
    // coefficient-form limbs that every one of its rows reads stay in L2 while they run
    const uint32_t poly = IOK == kIoModUp ? t / rw.count : t % rw.polys;
    const uint32_t slot = rw.first + (IOK == kIoModUp ? t % rw.count : t / rw.polys);
    const uint32_t pidx = row_prime(rw, slot);
    const uint32_t sig = threadIdx.x % S, lane = threadIdx.x / S;
    uint64_t *x = data + ((size_t)(poly * rw.slots + slot) << G::LOGN) + chunk * S;
    if (pidx == kNoPrime) return;  // ModUp: a limb of the digit itself
    const Limb<R> lb(pidx, false, tw, twd, pc);
    uint64_t a[G::E];
    if constexpr (IOK == kIoModUp) {
        const ModUpIO &mu = io.mu;
        __shared__ uint64_t sconv[16];
        const uint32_t b = slot / mu.LP, j = slot % mu.LP;
        const uint32_t s0 = b * mu.np, na = min(mu.np, mu.L - s0);
        if (threadIdx.x < na) sconv[threadIdx.x] = mu.conv[((size_t)b * mu.LP + j) * mu.np + threadIdx.x];
        __syncthreads();
        const PrimeConst p = pc[pidx];
        const uint64_t *y = mu.x + (((size_t)poly * mu.L + s0) << G::LOGN) + chunk * S;
#pragma unroll
        for (int m = 0; m < G::E; m++) {
            const size_t pos = sig + (size_t)G::M * (lane + m * G::E);
            a[m] = conv_sum(mu.sums, y + pos, sconv, na, G::LOGN, p);
        }
    } else if constexpr (IOK == kIoRescale) {
        const PrimeConst p = pc[pidx];
        const uint64_t *src = io.rs.last + ((size_t)poly << G::LOGN) + chunk * S;
#pragma unroll
        for (int m = 0; m < G::E; m++) a[m] = barrett({src[sig + (size_t)G::M * (lane + m * G::E)], 0}, p);
    } else if constexpr (IOK == kIoModDown) {
        __shared__ uint64_t sconv[16], svs[16];
        const uint32_t np = io.md.np, j = slot;
        if (threadIdx.x < np) sconv[threadIdx.x] = io.md.conv[(size_t)j * np + threadIdx.x];
        if (io.md.vrow && threadIdx.x < 16) svs[threadIdx.x] = io.md.vs[(size_t)j * 16 + threadIdx.x];
        __syncthreads();
        const PrimeConst p = pc[pidx];
        const uint64_t *z = io.md.acc + ((size_t)(poly * (rw.slots + np) + rw.slots) << G::LOGN) + chunk * S;
#pragma unroll
        for (int m = 0; m < G::E; m++) {
            const size_t pos = sig + (size_t)G::M * (lane + m * G::E);
            a[m] = conv_sum(io.md.sums, z + pos, sconv, np, G::LOGN, p);
        }
        if (io.md.vrow) {
            const uint8_t *vr = io.md.vrow + ((size_t)poly << G::LOGN) + chunk * S;
#pragma unroll
            for (int m = 0; m < G::E; m++) a[m] = sub_mod(a[m], svs[vr[sig + (size_t)G::M * (lane + m * G::E)] & 15], lb.q);
        }
    } else {
#pragma unroll
        for (int m = 0; m < G::E; m++) a[m] = x[sig + (size_t)G::M * (lane + m * G::E)];
    }
    if (IOK == kIoConverted) {
        // already doubles within about q/2 of zero, or in [0, q) for the integer families
    } else if (fam_has(FAM, kBfF64) && lb.mode == kBfF64) {  // [0, q) -> doubles for the FP64 butterflies
#pragma unroll
        for (int m = 0; m < G::E; m++) a[m] = as_bits(to_dbl(a[m]));
    } else if (fam_has(FAM, kBfF64R) && lb.mode == kBfF64R) {
#pragma unroll
        for (int m = 0; m < G::E; m++) a[m] = as_bits(to_dbl_centred(a[m], lb.q));
    }
    fwd_pass<R, FAM, false>(lb.mode, a, TwNatural{lb.t, 1}, lb.qd, lb.qinv, lb.w, lb.ws, 1, lb.q);
#pragma unroll
    for (int m = 0; m < G::E; m++) sm[(lane + m * G::E) * S + sig] = a[m];
    __syncthreads();
#pragma unroll
    for (int m = 0; m < G::E; m++) a[m] = sm[(lane * G::E + m) * S + sig];
    fwd_pass<R, FAM, false>(lb.mode, a, TwNatural{lb.t, G::E + lane}, lb.qd, lb.qinv, lb.w, lb.ws, G::E + lane, lb.q);
#pragma unroll
    for (int m = 0; m < G::E; m++) x[sig + (size_t)G::M * (lane * G::E + m)] = a[m];
}

// ---------------- forward, phase 2: blocks (global stages LOGM .. 2*LOGM-1), fully reduced output
// IOK = kIoRescale: instead of storing t = NTT(...) of row (poly, j), write (c_j - t) q_last^-1
// to io.rs.out; kIoModDown: write (acc_j - t) P^-1 (+ add) to io.md.out.  The words that the store
// combines are asked for (into L2) before the transform and read before its last barrier, and on the FP64
// rows t stays a double: the combination is one more twiddle-like product (27 limbs of 16 polynomials, ModDown:
// 0.294 ms with loads after the barrier and Shoup products, 0.189 ms so; rescale 0.189 and 0.129 ms).
template <int R, int S, int MINB, int IOK, int FAM>
__global__ void __launch_bounds__(Geo<R, S>::THREADS, MINB)
    fwd_blk(uint64_t *__restrict__ data, NttRows rw, const uint64_t *__restrict__ tw, const double *__restrict__ twd,
            const PrimeConst *__restrict__ pc, NttIO io) {
    using G = Geo<R, S>;
    __shared__ uint64_t sm[S * G::PAD_M];
    const uint32_t chunk = blockIdx.x % G::CHUNKS, t = blockIdx.x / G::CHUNKS;
    const uint32_t poly = t % rw.polys, slot = rw.first + t / rw.polys;
    const uint32_t pidx = row_prime(rw, slot);
    if (pidx == kNoPrime) return;
    const Limb<R> lb(pidx, false, tw, twd, pc);
    const uint32_t row = poly * rw.slots + slot;
    uint64_t *xc = data + ((size_t)row << G::LOGN) + (size_t)chunk * S * G::M;
    const uint32_t sig = threadIdx.x / G::E, lane = threadIdx.x % G::E;
    const uint32_t b = chunk * S + sig;
    uint64_t *x = xc + (size_t)sig * G::M;
    uint64_t *s = sm + sig * G::PAD_M;

    // where the store reads and writes: out = (in - t) mul (+ add[perm] add_mul)
    const size_t off = (size_t)chunk * S * G::M;
    const uint64_t *cin = nullptr, *mul = nullptr, *ad = nullptr, *amul = nullptr;
    const uint32_t *perm = nullptr;
    uint64_t *o = xc;
    if constexpr (IOK == kIoRescale) {
        cin = io.rs.in + (((size_t)poly * (rw.slots + 1) + slot) << G::LOGN) + off;
        o = io.rs.out + ((size_t)row << G::LOGN) + off;
        mul = io.rs.inv + 2 * slot;
    } else if constexpr (IOK == kIoModDown) {
        const ModDownIO &md = io.md;
        const uint32_t ct = poly / md.H, h = poly % md.H;
        cin = md.acc + (((size_t)poly * (rw.slots + md.np) + slot) << G::LOGN) + off;
        o = md.out + ct * md.out_ct + h * md.out_h + ((size_t)slot << G::LOGN) + off;
        mul = md.pinv + 2 * slot;
        if (h < md.n_add) {
            ad = md.add + ct * md.add_ct + h * md.add_h + ((size_t)slot << G::LOGN);
            if (h < md.n_perm && md.perm) perm = md.perm + off;
            if (md.add_mul) amul = md.add_mul + 2 * slot;
        }
    }
    if constexpr (IOK != kIoPlain) {
        constexpr uint32_t LINES = S * G::M / 16;  // 128-byte lines of the tile
        if (threadIdx.x < LINES) {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(cin + 16 * threadIdx.x));
            if (ad) {  // an automorphism maps aligned blocks of 32 words onto such blocks
                const size_t at = perm ? (__ldg(perm + (threadIdx.x / 2) * 32) & ~31u) + (threadIdx.x & 1) * 16
                                       : off + 16 * threadIdx.x;
                asm volatile("prefetch.global.L2 [%0];" ::"l"(ad + at));
            }
        }
    }

    uint64_t a[G::E];
#pragma unroll
    for (int m = 0; m < G::E; m++) a[m] = x[lane + m * G::E];
    fwd_pass<R, FAM, false>(lb.mode, a, TwNatural{lb.t, G::M + b}, lb.qd, lb.qinv, lb.w, lb.ws, G::M + b, lb.q);
#pragma unroll
    for (int m = 0; m < G::E; m++) s[padded(lane + m * G::E)] = a[m];
    __syncthreads();
#pragma unroll
    for (int m = 0; m < G::E; m++) a[m] = s[padded(lane * G::E + m)];
    fwd_pass<R, FAM, true>(lb.mode, a, TwLane<R>(lb.t, b, lane), lb.qd, lb.qinv, lb.w, lb.ws,
                           ((G::M + b) << R) + lane, lb.q);
    const bool fp = fam_fp(FAM) && (!fam_int(FAM) || lb.fp());
    if (fp) {
        if constexpr (IOK == kIoPlain) {
#pragma unroll
            for (int m = 0; m < G::E; m++) s[padded(lane * G::E + m)] = dbl_mod(as_dbl(a[m]), lb.qd, lb.qinv);
        } else {  // |t| < 11 q (kBfF64), centred (kBfF64R): in - t stays inside mul_dbl's range
#pragma unroll
            for (int m = 0; m < G::E; m++)
                s[padded(lane * G::E + m)] =
                    lb.mode == kBfF64 ? a[m] : as_bits(dbl_centre(as_dbl(a[m]), lb.qd, lb.qinv));
        }
    } else if (fam_has(FAM, kBfGrow) && lb.mode == kBfGrow) {
        const PrimeConst p = pc[pidx];
#pragma unroll
        for (int m = 0; m < G::E; m++) s[padded(lane * G::E + m)] = reduce_small(a[m], p);  // < 68q -> [0, q)
    } else {
        const uint64_t q2 = 2 * lb.q;
#pragma unroll
        for (int m = 0; m < G::E; m++) s[padded(lane * G::E + m)] = csub(csub(a[m], q2), lb.q);
    }
    auto at = [&](int i) { return threadIdx.x + i * G::THREADS; };
    auto result = [&](int i) { return sm[(at(i) / G::M) * G::PAD_M + padded(at(i) % G::M)]; };
    if constexpr (IOK == kIoPlain) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < G::E; i++) xc[at(i)] = result(i);
    } else {
        const uint64_t q = lb.q;
        uint64_t v[G::E];
#pragma unroll
        for (int i = 0; i < G::E; i++) v[i] = cin[at(i)];
        __syncthreads();
        if (fp) {
            const double w = to_dbl_centred(mul[0], q);
#pragma unroll
            for (int i = 0; i < G::E; i++)
                v[i] = as_bits(mul_dbl(__dsub_rn(to_dbl(v[i]), as_dbl(result(i))), w, lb.qd, lb.qinv));
            if (!ad) {
#pragma unroll
                for (int i = 0; i < G::E; i++) o[at(i)] = dbl_canon(as_dbl(v[i]), lb.qd);
            } else if (amul) {
                const double aw = to_dbl_centred(amul[0], q);
#pragma unroll
                for (int i = 0; i < G::E; i++) {
                    const double u = mul_dbl(to_dbl(ad[perm ? __ldg(perm + at(i)) : off + at(i)]), aw, lb.qd, lb.qinv);
                    o[at(i)] = dbl_mod(__dadd_rn(as_dbl(v[i]), u), lb.qd, lb.qinv);
                }
            } else {
#pragma unroll
                for (int i = 0; i < G::E; i++)
                    o[at(i)] = add_mod(dbl_canon(as_dbl(v[i]), lb.qd), ad[perm ? __ldg(perm + at(i)) : off + at(i)], q);
            }
        } else {
            const uint64_t w = mul[0], ws = mul[1], aw = amul ? amul[0] : 0, aws = amul ? amul[1] : 0;
#pragma unroll
            for (int i = 0; i < G::E; i++) {
                uint64_t r = shoup(sub_mod(v[i], result(i), q), w, ws, q);
                if (ad) {
                    const uint64_t u = ad[perm ? __ldg(perm + at(i)) : off + at(i)];
                    r = add_mod(r, amul ? shoup(u, aw, aws, q) : u, q);
                }
                o[at(i)] = r;
            }
        }
    }
}

// ---------------- inverse, phase 1: blocks (global stages 2*LOGM-1 .. LOGM)
// reads polynomial p's limbs at src + p src_stride (data's own rows, or another buffer's)
template <int R, int S, int MINB, int FAM>
__global__ void __launch_bounds__(Geo<R, S>::THREADS, MINB)
    inv_blk(uint64_t *data, const uint64_t *src, size_t src_stride, NttRows rw,
            const uint64_t *__restrict__ tw, const double *__restrict__ twd, const PrimeConst *__restrict__ pc) {
    using G = Geo<R, S>;
    __shared__ uint64_t sm[S * G::PAD_M];
    const uint32_t chunk = blockIdx.x % G::CHUNKS, t = blockIdx.x / G::CHUNKS;
    const uint32_t poly = t % rw.polys, slot = rw.first + t / rw.polys;
    const Limb<R> lb(row_prime(rw, slot), true, tw, twd, pc);
    const size_t off = (size_t)chunk * S * G::M;
    uint64_t *xc = data + ((size_t)(poly * rw.slots + slot) << G::LOGN) + off;
    const uint64_t *in = src + poly * src_stride + ((size_t)slot << G::LOGN) + off;
    const uint32_t sig = threadIdx.x / G::E, lane = threadIdx.x % G::E;
    const uint32_t b = chunk * S + sig;
    uint64_t *s = sm + sig * G::PAD_M;

#pragma unroll
    for (int i = 0; i < G::E; i++) {
        uint32_t e = threadIdx.x + i * G::THREADS;
        sm[(e / G::M) * G::PAD_M + padded(e % G::M)] = in[e];
    }
    __syncthreads();
    uint64_t a[G::E];
#pragma unroll
    for (int m = 0; m < G::E; m++) a[m] = s[padded(lane * G::E + m)];
    if (fam_fp(FAM) && (!fam_int(FAM) || lb.fp())) {
#pragma unroll
        for (int m = 0; m < G::E; m++) a[m] = as_bits(to_dbl(a[m]));
    }
    inv_pass<R, FAM, false>(lb.mode, a, TwLane<R>(lb.t, b, lane), lb.qd, lb.qinv, lb.w, lb.ws,
                            ((G::M + b) << R) + lane, lb.q);
#pragma unroll
    for (int m = 0; m < G::E; m++) s[padded(lane * G::E + m)] = a[m];
    __syncthreads();
#pragma unroll
    for (int m = 0; m < G::E; m++) a[m] = s[padded(lane + m * G::E)];
    inv_pass<R, FAM, false>(lb.mode, a, TwNatural{lb.t, G::M + b}, lb.qd, lb.qinv, lb.w, lb.ws, G::M + b, lb.q);
    uint64_t *x = xc + (size_t)sig * G::M;
#pragma unroll
    for (int m = 0; m < G::E; m++) x[lane + m * G::E] = a[m];
}

// ---------------- inverse, phase 2: columns (global stages LOGM-1 .. 0) with the folded scale
template <int R, int S, int MINB, int FAM>
__global__ void __launch_bounds__(Geo<R, S>::THREADS, MINB)
    inv_col(uint64_t *__restrict__ data, NttRows rw, const uint64_t *__restrict__ tw, const double *__restrict__ twd,
            const PrimeConst *__restrict__ pc, const uint64_t *__restrict__ scale, int scale_by_prime) {
    using G = Geo<R, S>;
    __shared__ uint64_t sm[G::M * S];
    const uint32_t chunk = blockIdx.x % G::CHUNKS, t = blockIdx.x / G::CHUNKS;
    const uint32_t poly = t % rw.polys, slot = rw.first + t / rw.polys;
    const uint32_t pidx = row_prime(rw, slot);
    const Limb<R> lb(pidx, true, tw, twd, pc);
    const uint64_t q = lb.q;
    const uint64_t *sc = scale + 4 * (scale_by_prime ? pidx : slot - rw.first);
    uint64_t *x = data + ((size_t)(poly * rw.slots + slot) << G::LOGN) + chunk * S;
    const uint32_t sig = threadIdx.x % S, lane = threadIdx.x / S;

    uint64_t a[G::E];
#pragma unroll
    for (int m = 0; m < G::E; m++) a[m] = x[sig + (size_t)G::M * (lane * G::E + m)];
    inv_pass<R, FAM, false>(lb.mode, a, TwNatural{lb.t, G::E + lane}, lb.qd, lb.qinv, lb.w, lb.ws, G::E + lane, q);
#pragma unroll
    for (int m = 0; m < G::E; m++) sm[(lane * G::E + m) * S + sig] = a[m];
    __syncthreads();
#pragma unroll
    for (int m = 0; m < G::E; m++) a[m] = sm[(lane + m * G::E) * S + sig];
    inv_pass<R, FAM, true>(lb.mode, a, TwNatural{lb.t, 1}, lb.qd, lb.qinv, lb.w, lb.ws, 1, q);
    if (fam_fp(FAM) && (!fam_int(FAM) || lb.fp())) {
        // the last stage and the scale: products of u +- v, each below q in magnitude
        const double c0 = to_dbl_centred(sc[0], q), c1 = to_dbl_centred(sc[2], q);
#pragma unroll
        for (int m = 0; m < G::E / 2; m++) {
            const double u = as_dbl(a[m]), v = as_dbl(a[m + G::E / 2]);
            a[m] = dbl_canon(mul_dbl(__dadd_rn(u, v), c0, lb.qd, lb.qinv), lb.qd);
            a[m + G::E / 2] = dbl_canon(mul_dbl(__dsub_rn(u, v), c1, lb.qd, lb.qinv), lb.qd);
        }
    } else {
        // values in [0, 4q) (grow) or [0, 2q) (Harvey)
        const uint64_t c0 = sc[0], c0s = sc[1], c1 = sc[2], c1s = sc[3], q2 = (lb.mode != kBfHarvey ? 4 : 2) * q;
#pragma unroll
        for (int m = 0; m < G::E / 2; m++) {
            uint64_t u = a[m], v = a[m + G::E / 2];
            a[m] = shoup(u + v, c0, c0s, q);
            a[m + G::E / 2] = shoup(u - v + q2, c1, c1s, q);
        }
    }
#pragma unroll
    for (int m = 0; m < G::E; m++) x[sig + (size_t)G::M * (lane + m * G::E)] = a[m];
}

// ---------------- launches

// one inverse transform: rows of `data`, read from src (polynomials src_stride words apart); scale:
// [rw.count][4] (c, c', c psi^-(N/2), its companion), or null for the plain N^-1 of each prime
struct InvArgs {
    uint64_t *data;
    const uint64_t *src;
    size_t src_stride;
    const uint64_t *scale;
};

template <int R, int S, int MINB, int IOK, int FAM>
void launch_fwd_v(const Context &c, uint64_t *data, const NttRows &rw, cudaStream_t st, const NttIO &io) {
    using G = Geo<R, S>;
    dim3 grid(rw.polys * rw.count * G::CHUNKS);
    constexpr int BLK = IOK == kIoModUp ? kIoPlain : IOK;  // ModUp's block phase is a plain one
    SHM_LAUNCHED(1);
    // rows converted by conv_rows: the plain column phase, whose input is in the butterflies' form
    if constexpr (IOK == kIoModUp || IOK == kIoModDown) {
        if (io.converted) {
            fwd_col<R, S, MINB, kIoConverted, FAM><<<grid, G::THREADS, 0, st>>>(data, rw, c.tw, c.twd, c.pc, io);
        } else {
            // a conversion in the loads (more than eight limbs) waits for them longer than the 24 warps an SM of
            // 8 x 6 cover: 18 limbs in digits of nine, eight key switches at 50 bits 1.35 ms with 8 x 6, 1.11 with
            // 16 x 4 here; one at 58 bits 366 and 299 us
            constexpr int SC = MINB == 6 ? 16 : S, MC = MINB == 6 ? 4 : MINB;
            using GC = Geo<R, SC>;
            const dim3 cg(rw.polys * rw.count * GC::CHUNKS);
            fwd_col<R, SC, MC, IOK, FAM><<<cg, GC::THREADS, 0, st>>>(data, rw, c.tw, c.twd, c.pc, io);
        }
    } else {
        fwd_col<R, S, MINB, IOK, FAM><<<grid, G::THREADS, 0, st>>>(data, rw, c.tw, c.twd, c.pc, io);
    }
    SHM_LAUNCHED(1);
    fwd_blk<R, S, MINB, BLK, FAM><<<grid, G::THREADS, 0, st>>>(data, rw, c.tw, c.twd, c.pc, io);
}

template <int R, int S, int MINB, int FAM>
void launch_inv_v(const Context &c, const InvArgs &v, const NttRows &rw, cudaStream_t st) {
    using G = Geo<R, S>;
    dim3 grid(rw.polys * rw.count * G::CHUNKS);
    SHM_LAUNCHED(1);
    inv_blk<R, S, MINB, FAM><<<grid, G::THREADS, 0, st>>>(v.data, v.src, v.src_stride, rw, c.tw, c.twd, c.pc);
    SHM_LAUNCHED(1);
    inv_col<R, S, MINB, FAM><<<grid, G::THREADS, 0, st>>>(v.data, rw, c.tw, c.twd, c.pc,
                                                          v.scale ? v.scale : c.inv_scale_plain, v.scale ? 0 : 1);
}

// the tile variants of kNttVariants (ntt.cuh), selected per context by c.ntt_variant
template <int R, int IOK, int FAM>
void launch_fwd_f(const Context &c, uint64_t *data, const NttRows &rw, cudaStream_t st, const NttIO &io) {
    switch (c.ntt_variant) {
        case 1: launch_fwd_v<R, 16, 3, IOK, FAM>(c, data, rw, st, io); break;
        case 2: launch_fwd_v<R, 8, 8, IOK, FAM>(c, data, rw, st, io); break;
        case 3: launch_fwd_v<R, 8, 6, IOK, FAM>(c, data, rw, st, io); break;
        default: launch_fwd_v<R, 16, 4, IOK, FAM>(c, data, rw, st, io); break;
    }
}

// A forward transform of the rows of `data` in the butterfly families FAM and the ring R; kind: the load and
// store transforms
template <int R, int FAM>
void launch_fwd(const Context &c, int kind, uint64_t *data, const NttRows &rw, cudaStream_t st, const NttIO &io) {
    switch (kind) {
        case kIoPlain: launch_fwd_f<R, kIoPlain, FAM>(c, data, rw, st, io); break;
        case kIoRescale: launch_fwd_f<R, kIoRescale, FAM>(c, data, rw, st, io); break;
        case kIoModDown: launch_fwd_f<R, kIoModDown, FAM>(c, data, rw, st, io); break;
        default: launch_fwd_f<R, kIoModUp, FAM>(c, data, rw, st, io); break;
    }
}

template <int R, int FAM>
void launch_inv(const Context &c, const InvArgs &v, const NttRows &rw, cudaStream_t st) {
    switch (c.ntt_variant) {
        case 1: launch_inv_v<R, 16, 3, FAM>(c, v, rw, st); break;
        case 2: launch_inv_v<R, 8, 8, FAM>(c, v, rw, st); break;
        case 3: launch_inv_v<R, 8, 6, FAM>(c, v, rw, st); break;
        default: launch_inv_v<R, 16, 4, FAM>(c, v, rw, st); break;
    }
}

}  // namespace shm

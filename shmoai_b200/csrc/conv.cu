// Base conversions on the tensor cores (ModUp's digits, ModDown's special-prime limbs).
//
// A conversion is a small contraction: row j of a set is sum_i y_i c_ij mod q_j over the set's limbs.
// With y_i = sum_b y_ib 2^(8b) and the constants c_ijb = c_ij 2^(8b) mod q_j cut into bytes too,
//   sum_i y_i c_ij = sum_o 2^(8o) D_o (mod q_j),   D_o = sum_(i,b) y_ib (c_ijb)_o:
// per coefficient a product of its 8 na <= 64 limb bytes (the MMA's A rows are the limbs' 64-bit words
// as they lie in memory) with a 64 x 8 byte matrix per row j, exact in s32 (below 64 255^2 < 2^22).
// The eight sums of a coefficient come back from TMEM to the thread of that coefficient, are packed
// into V = high 2^32 + low (< 2^14 q, as every c_ijb < q), and Q = round(high 2^32 / q) from the FP64
// pipe leaves V - Q q within q/2 + 2^32 of zero: the double the FP64 butterflies take, written as such
// (integer families add q to a negative one).
//
// What bounds it: issue (47 instructions a coefficient and row, a third of them the wait, address and
// constant handling of a step) at 16 warps per SM and 128 registers, 0.53 of the measured copy rate.  On the CUDA cores the same sum
// of five terms took 20 wide multiplies (which issue at a quarter of the rate), a 128-bit fold and a Barrett
// reduction inside the NTT's column phase, where each row also re-read the set's limbs from L2: 190 issued
// instructions per coefficient against 55 for the plain column phase.  Eight ciphertexts at 27 limbs (48
// digits of five limbs to 27 rows each): column phase 0.97 ms with the conversion in its loads; 0.23 ms
// here and 0.285 ms for the plain column phase.  As part of the column kernel (the limbs resident in TMEM or
// shared memory, a row at a time) it took 0.63 ms: one CTA per SM left the butterflies without warps.
#include <algorithm>

#include "core.hpp"
#include "tcgen05.cuh"

namespace shm {

namespace {

constexpr uint32_t kT = 128;         // threads of a CTA: an MMA row each
constexpr uint32_t kPer = 2;         // MMA tiles, and coefficients of a thread, at a time
constexpr uint32_t kTile = kT * kPer;
constexpr uint32_t kRows = 4;        // rows of a step: N = 32 byte columns
constexpr uint32_t kCols = 128;      // TMEM columns of a CTA: A of this and the next tile (64), one step's sums (64)
constexpr uint32_t kRowBytes = 512;  // a row's constants

struct RowConst {
    uint64_t neg_q;  // 2^64 - q
    double k32;      // 2^32 / q
};

// V = sum_o w_o 2^(8 o) in words: high 2^32 + low, high = h1 2^32 + h0 < 2^48.  k16 = 2^16 as a register:
// the two wide multiply-adds stay such (as shifts and adds with carries they are eight operations)
__device__ __forceinline__ void pack(const uint32_t *w, uint32_t k16, uint32_t &low, uint32_t &h0, uint32_t &h1) {
    const uint64_t a = (uint64_t)(w[2] + (w[3] << 8)) * k16 + (w[0] + (w[1] << 8));
    low = (uint32_t)a;
    const uint64_t b = (uint64_t)(w[6] + (w[7] << 8)) * k16 + (w[4] + (w[5] << 8) + (uint32_t)(a >> 32));
    h0 = (uint32_t)b;
    h1 = (uint32_t)(b >> 32);
}

// {lo, hi} + a b mod 2^64
__device__ __forceinline__ uint64_t mad_low(uint32_t a, uint64_t b, uint32_t lo, uint32_t hi) {
    uint64_t r = (uint64_t)hi << 32 | lo;
    asm("{\n\t.reg .u32 l, h, b0, b1;\n\t"
        "mov.b64 {b0, b1}, %2;\n\t"
        "mad.wide.u32 %0, %1, b0, %0;\n\t"
        "mov.b64 {l, h}, %0;\n\t"
        "mad.lo.u32 h, %1, b1, h;\n\t"
        "mov.b64 %0, {l, h};\n\t}"
        : "+l"(r)
        : "r"(a), "l"(b));
    return r;
}

// Grid: sets x coefficient blocks of `tiles` tiles of kTile.  Dynamic shared memory: the rows' constants
// (steps of kRows rows), then their RowConst and output rows.  A CTA goes through (tile, step) pairs: wait
// for the step's sums, read them, issue the next step's MMAs once all four warps have read, convert and
// store; the next tile's limb words go to the other A buffer during a tile's first step.  A thread whose wait runs
// out stores nothing from then on and sets *fault; the issuing thread issues no more, and its MMAs in flight are
// waited for (with a bound too) before the TMEM is freed.
// ALL_FP: every row's butterflies run on doubles (every prime below 2^51).  LIMITED: `limit` polls a wait instead
// of kSpinLimit (a run-time bound of every wait costs 2 % of the kernel).
template <bool ALL_FP, bool LIMITED>
__global__ void __launch_bounds__(kT, 4) conv_kernel(ConvIO io, uint32_t log_n, uint32_t tiles, uint32_t k16,
                                                     const PrimeConst *__restrict__ pc, int *__restrict__ fault, int limit) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t full, drained;
    __shared__ uint32_t tmem_base;
    const uint32_t tid = threadIdx.x, warp = tid / 32;
    const uint32_t blocks = (1u << log_n) / (kTile * tiles), set = blockIdx.x / blocks, blk = blockIdx.x % blocks;
    const uint32_t ct = set / io.per, dig = set % io.per, l0 = dig * io.na, na = min(io.na, io.total - l0);
    const uint32_t own = io.skip_own ? na : 0, rows = io.rows - own;  // rows l0 .. l0 + na - 1 are left alone
    const uint32_t steps = (rows + kRows - 1) / kRows;
    const uint32_t nk = na + (io.vrow ? 1 : 0) > 4 ? 2 : 1;  // K = 32 slices
    RowConst *rc = reinterpret_cast<RowConst *>(smem + (size_t)steps * kRows * kRowBytes);
    uint32_t *rj = reinterpret_cast<uint32_t *>(rc + steps * kRows);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_base)),
                     "r"(kCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&full)));
        asm volatile("fence.mbarrier_init.release.cluster;\n");
    }
    // constants: row r of the set at r 512, so rows 8 k .. 8 k + 7 of an MMA's B operand are one block
    for (uint32_t e = tid; e < rows * (kRowBytes / 16); e += kT) {
        const uint32_t r = e / (kRowBytes / 16), j = own && r >= l0 ? r + own : r;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(smem_u32(smem + e * 16)),
                     "l"(io.bytes + ((size_t)dig * io.rows + j) * kRowBytes + e % (kRowBytes / 16) * 16)
                     : "memory");
    }
    for (uint32_t r = tid; r < rows; r += kT) {
        const uint32_t j = own && r >= l0 ? r + own : r;
        const PrimeConst p = pc[io.prime(j)];
        rc[r] = RowConst{0 - p.q, __dmul_rn(4294967296.0, p.qinv)};
        rj[r] = j;
    }
    const uint64_t *src = io.src + ct * io.src_ct + ((size_t)l0 << log_n) + (size_t)blk * tiles * kTile + tid;
    const uint8_t *vr = io.vrow ? io.vrow + ((size_t)set << log_n) + (size_t)blk * tiles * kTile + tid : nullptr;
    uint64_t v[kPer][kConvSlots];
    auto load = [&](uint32_t t) {  // this thread's coefficients of tile t: limb words, the overflow count, zeros
#pragma unroll
        for (uint32_t e = 0; e < kPer; e++) {
            const size_t pos = t * kTile + e * kT;
#pragma unroll
            for (uint32_t i = 0; i < kConvSlots; i++) v[e][i] = i < na ? __ldg(src + ((size_t)i << log_n) + pos) : 0;
            if (vr) {
                const uint64_t over = vr[pos];
#pragma unroll
                for (uint32_t i = 0; i < kConvSlots; i++)
                    if (i == na) v[e][i] = over;
            }
        }
    };
    auto store_a = [&](uint32_t addr) {
#pragma unroll
        for (uint32_t e = 0; e < kPer; e++) {
            const uint64_t *w = v[e];
            asm volatile(
                "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
                "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(addr + e * 16),
                "r"((uint32_t)w[0]), "r"((uint32_t)(w[0] >> 32)), "r"((uint32_t)w[1]), "r"((uint32_t)(w[1] >> 32)),
                "r"((uint32_t)w[2]), "r"((uint32_t)(w[2] >> 32)), "r"((uint32_t)w[3]), "r"((uint32_t)(w[3] >> 32)),
                "r"((uint32_t)w[4]), "r"((uint32_t)(w[4] >> 32)), "r"((uint32_t)w[5]), "r"((uint32_t)(w[5] >> 32)),
                "r"((uint32_t)w[6]), "r"((uint32_t)(w[6] >> 32)), "r"((uint32_t)w[7]), "r"((uint32_t)(w[7] >> 32))
                : "memory");
        }
        asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
    };
    load(0);
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    const uint32_t tmem = tmem_base, tq = tmem + (warp << 21);  // this warp's 32 lanes
    // s32 accumulators, A (TMEM) and B unsigned bytes, K-major, N = 32, M = 128
    const uint32_t idesc = (2u << 4) | ((kRows * 8 >> 3) << 17) | ((128u >> 4) << 24);
    const uint32_t bar = smem_u32(&full), b_addr = smem_u32(smem);
    bool ok = true;
    auto issue = [&](uint32_t t, uint32_t c) {  // the MMAs of tile t, step c
        if (tid == 0 && ok) {
#pragma unroll
            for (uint32_t e = 0; e < kPer; e++)
                for (uint32_t k = 0; k < nk; k++)
                    asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(tmem + 64 + e * 32),
                    "r"(tmem + (t & 1) * 32 + e * 16 + k * 8), "l"(smem_desc(b_addr + c * (kRows * kRowBytes) + k * 256)),
                    "r"(idesc), "r"(k));
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar));
        }
    };
    store_a(tq);
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    issue(0, 0);
    if (tiles > 1) load(1);

    uint32_t phase = 0;
    const uint32_t row_bytes = 8u << log_n;
    char *out = reinterpret_cast<char *>(io.out + (((size_t)set * io.rows) << log_n) + (size_t)blk * tiles * kTile + tid);
    for (uint32_t t = 0; t < tiles; t++, out += kTile * 8) {
        for (uint32_t c = 0; c < steps; c++) {
            if (ok && !mbar_wait(bar, phase, LIMITED ? limit : kSpinLimit)) ok = false;
            phase ^= 1;
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;\n");
            uint32_t d[kPer][kRows][8];
#pragma unroll
            for (uint32_t e = 0; e < kPer; e++)
#pragma unroll
                for (uint32_t h = 0; h < kRows; h++)
                    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                                 : "=r"(d[e][h][0]), "=r"(d[e][h][1]), "=r"(d[e][h][2]), "=r"(d[e][h][3]),
                                   "=r"(d[e][h][4]), "=r"(d[e][h][5]), "=r"(d[e][h][6]), "=r"(d[e][h][7])
                                 : "r"(tq + 64 + e * 32 + h * 8));
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
            if (c == 0 && t + 1 < tiles) store_a(tq + ((t + 1) & 1) * 32);  // its last reader was tile t - 1
            asm volatile("tcgen05.fence::before_thread_sync;\n");
            __syncthreads();  // all sums have been read
            asm volatile("tcgen05.fence::after_thread_sync;\n");
            if (c + 1 < steps) issue(t, c + 1);
            else if (t + 1 < tiles) issue(t + 1, 0);
            if (c == 0 && t + 2 < tiles) load(t + 2);
            if (!ok) continue;
            const RowConst *kc = rc + c * kRows;
            const uint32_t *jc = rj + c * kRows;
#pragma unroll
            for (uint32_t h = 0; h < kRows; h++) {
                if (c * kRows + h >= rows) break;
                const RowConst k = kc[h];
                uint64_t *o = reinterpret_cast<uint64_t *>(out + (uint64_t)jc[h] * row_bytes);
#pragma unroll
                for (uint32_t e = 0; e < kPer; e++) {
                    uint32_t low, h0, h1;
                    pack(d[e][h], k16, low, h0, h1);
                    const double hd = __dsub_rn(__hiloint2double(h1 | 0x43300000, h0), kTwo52);
                    const uint32_t Q = (uint32_t)__double2loint(__fma_rn(hd, k.k32, kTwo52));
                    uint64_t x;  // V - Q q
                    if (ALL_FP || 0 - k.neg_q < kF64CentreLimit) {
                        x = mad_low(Q, k.neg_q, low, h0 + 0x43380000u);  // its bits plus those of 1.5 2^52
                        x = as_bits(__dsub_rn(as_dbl(x), kMagic));
                    } else {
                        x = mad_low(Q, k.neg_q, low, h0);
                        x -= (uint64_t)((int64_t)x >> 63) & k.neg_q;
                    }
                    o[e * kT] = x;
                }
            }
        }
    }
    if (!ok) {
        *fault = 1;
        if (tid == 0) {  // the MMAs in flight
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&drained)));
            asm volatile("fence.mbarrier_init.release.cluster;\n");
            asm volatile("fence.proxy.async.shared::cta;\n");
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                smem_u32(&drained)));
            mbar_wait(smem_u32(&drained), 0);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kCols));
}

}  // namespace

// Tiles per CTA: the constants (20 KB for 40 rows) are read once per CTA, so as many as leave a CTA
// for each of the four places per SM four times over.
void conv_rows(const Context &c, const ConvIO &io, cudaStream_t st) {
    if (io.sets == 0 || io.rows == 0) return;
    const uint32_t all = c.n / kTile;
    uint32_t tiles = 1;
    while (tiles < 32 && tiles * 2 <= all && (uint64_t)io.sets * (all / (tiles * 2)) >= 16ull * c.sms) tiles *= 2;
    // the last step's rows past the end are in the buffer, unwritten: their sums are not used
    const size_t smem = (io.rows + kRows - 1) / kRows * kRows * (kRowBytes + sizeof(RowConst) + sizeof(uint32_t));
    const bool fp = c.ntt_families == kFamSmall, limited = c.wait_limit != kSpinLimit;
    const auto f = limited ? (fp ? conv_kernel<true, true> : conv_kernel<false, true>)
                           : (fp ? conv_kernel<true, false> : conv_kernel<false, false>);
    static std::atomic<uint64_t> ready{0};  // a bit per device: the attribute belongs to the device's module
    const uint64_t bit = 1ull << (c.device & 63);
    if (!(ready.load(std::memory_order_acquire) & bit)) {
        for (const auto k : {conv_kernel<true, true>, conv_kernel<false, true>, conv_kernel<true, false>,
                             conv_kernel<false, false>})
            SHM_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        ready.fetch_or(bit, std::memory_order_release);
    }
    SHM_LAUNCHED(1);
    const dim3 grid(io.sets * (all / tiles));
    f<<<grid, kT, smem, st>>>(io, c.log_n, tiles, 65536u, c.pc, c.fault_dev, c.wait_limit);
    SHM_CUDA(cudaGetLastError());
}

}  // namespace shm

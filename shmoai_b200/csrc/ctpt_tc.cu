// Rotation-free ct-pt matmul on the INT8 tensor cores (tcgen05.mma kind::i8), exact.
//
// Y[o][r] = sum_i X[i][r] * W[i][o] mod q_limb(r): X rows r of the n_in input
// ciphertexts (2 L N residues each), W the signed integer weights.  This is the
// reference's multiply_plain + add_inplace loop over constant plaintexts
// (src/include/source/matrix_mul/Ct_pt_matrix_mul.cuh:112-158) computed as one
// dense contraction.
//
// Exactness by a small-modulus residue system: the integer S = sum_i x_i w_i
// (|S| <= (q_l - 1) max_o sum_i |w_io|) is computed modulo T pairwise-coprime moduli
// m_t <= 251 whose product exceeds 2.02 |S|, each as an int8 GEMM with balanced
// residues in [-125, 125] (|acc| < n_in * 125^2 < 2^31), then rebuilt by the CRT:
//   S = sum_t r_t c_t - v M,  c_t = (M/m_t) [(M/m_t)^-1]_{m_t},  v = round(sum_t r_t inv_t / m_t),
// and reduced mod q_l with per-limb constants.  T GEMMs replace the 35 byte-slice
// products of a positional split; T is chosen per limb (a smaller prime needs fewer moduli)
// and each pass of columns runs with the largest T of its limbs.
//
// Pipeline per pass of columns: X residue planes [T][R][K] and W residue planes [T][N][K]
// (both K-major) -> tcgen05 GEMMs (weights as the M = 128 side, 256 X columns as N, s32
// accumulators in TMEM; operands by TMA where the X tile fits in shared memory) ->
// epilogue tcgen05.ld, acc mod m_t -> uint8 residue planes -> CRT kernel.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <cmath>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "core.hpp"
#include "host_math.hpp"
#include "tcgen05.cuh"  // kKB: K bytes per stage (two k32 MMAs)

namespace shm {

namespace {

constexpr int kMaxMods = 20;
constexpr uint32_t kBM = 128;   // outputs per tile (MMA M: A = the weight residues)
constexpr uint32_t kBN = 256;   // X columns per tile (MMA N: B = the X residues)
constexpr int kStages = 4;
constexpr uint32_t kStageA = kBM * kKB;  // 8 KB
constexpr uint32_t kStageB = kBN * kKB;  // 16 KB
constexpr uint32_t kSmem = kStages * (kStageA + kStageB) + 1024;
constexpr uint32_t kThreads = 256;  // two warpgroups: loads shared, epilogue split by output columns

// The constants of every candidate modulus, and the CRT fractions for every modulus count T
// (M = m_0 .. m_{T-1}): the table does not depend on the call, so concurrent calls that
// write it write the same bytes; each kernel takes its T as an argument.
struct ModTab {
    uint32_t m[kMaxMods];
    uint32_t fracq[kMaxMods + 1][kMaxMods];  // [T][t]: round(2^19 [(M/m_t)^-1]_{m_t} / m_t)
    uint32_t c24[kMaxMods];  // 2^20 mod m_t
    uint32_t c48[kMaxMods];  // 2^40 mod m_t
    uint32_t magic[kMaxMods];  // ceil(2^32 / m_t)
    int rnd[kMaxMods];         // round(2^32 / m_t)
    uint32_t vbase[kMaxMods + 1];  // [T]: the CRT's v before the residues (crt_kernel)
    double inv[kMaxMods];    // 1 / m_t
};

__constant__ ModTab c_mods;

// ---------------------------------------------------------------- residues
__device__ __forceinline__ int8_t balanced(uint32_t r, uint32_t m) { return (int8_t)(r > m / 2 ? (int)r - (int)m : (int)r); }

// x mod m_t for x < 2^61 in 32-bit arithmetic: x = a 2^40 + b 2^20 + d (a < 2^21, b, d < 2^20)
// folds to s = a (2^40 mod m) + b (2^20 mod m) + d < 2^30; the quotient
// umulhi(s, ceil(2^32 / m)) is floor(s / m) or one more.
__device__ __forceinline__ uint32_t mod_small(uint64_t x, uint32_t t) {
    const uint32_t m = c_mods.m[t];
    const uint32_t a = (uint32_t)(x >> 40), b = (uint32_t)(x >> 20) & 0xFFFFF, d = (uint32_t)x & 0xFFFFF;
    const uint32_t s = a * c_mods.c48[t] + b * c_mods.c24[t] + d;
    int r = (int)(s - __umulhi(s, c_mods.magic[t]) * m);
    return (uint32_t)(r < 0 ? r + (int)m : r);
}

// The residue planes of the products hold a balanced residue of S mod m_t plus 128, a byte.
//
// An accumulator's residue in [-127, 127] for |a| <= kAccSmall (n_in up to 4,160 inputs): q = round(a / m)
// from one wide multiply-add with round(2^32 / m) (|q - a / m| <= 1/2 + |a| 2^-33), so |a - q m| <= m / 2 +
// m |a| 2^-33 < 127.5 with no correction; its low byte is the residue.  Two operations an accumulator and
// none on the conversion pipe: an int -> float -> int quotient (16 conversions a clock per SM) held a 128 x 256
// tile's epilogue to 2.1 us at least, the tile's MMAs at K = 768 to 1.6 us.
constexpr uint64_t kAccSmall = 65000000;
__device__ __forceinline__ uint32_t acc_residue(int a, int rnd, uint32_t m) {
    const int64_t p = (int64_t)a * rnd + 0x80000000ll;
    return (uint32_t)a - (uint32_t)(p >> 32) * m;
}

// any int32 accumulator: a + m * 2^24 (a multiple of m above 2^31, the moduli being > 128) is
// non-negative and below 2^33, then the 32-bit fold above
__device__ __forceinline__ uint32_t acc_residue_any(int a, uint32_t t) {
    const uint32_t r = mod_small((uint64_t)((int64_t)a + ((int64_t)c_mods.m[t] << 24)), t);
    return (uint32_t)(int)balanced(r, c_mods.m[t]);
}

// The balanced residue of x mod m_t (in (-m/2, m/2), m odd) for x < 2^51 given as the exact double
// xd and its low word xlo: q = round(x / m) from fma(xd, 1/m, 1.5 2^52) (the pre-rounding value is
// within (x / m) 2^-53 < 0.25 / m of x / m, and x / m lies at least 0.5 / m from a half-integer,
// so q is the nearest integer).  The fma's result 1.5 2^52 + q carries q in the low bits of its
// mantissa (2^51 is a multiple of 2^32), so (x - q m) mod 2^32 = xlo - q_lo m, whose low byte is
// the two's complement of the residue: one FP64 multiply-add and one integer multiply-add.
__device__ __forceinline__ uint32_t balanced_f64(double xd, uint32_t xlo, uint32_t t) {
    const double magic = 6755399441055744.0;  // 1.5 * 2^52
    const uint32_t q = (uint32_t)__double2loint(__fma_rn(xd, c_mods.inv[t], magic));
    return xlo - q * c_mods.m[t];
}

// the low bytes of four words as one word
__device__ __forceinline__ uint32_t pack_low_bytes(uint32_t b0, uint32_t b1, uint32_t b2, uint32_t b3) {
    return __byte_perm(__byte_perm(b0, b1, 0x0040), __byte_perm(b2, b3, 0x0040), 0x5410);
}

// four accumulators as four bytes of the plane
__device__ __forceinline__ uint32_t acc_bytes(const uint32_t *v, uint32_t t, int small) {
    uint32_t r[4];
    if (small) {
        const int rnd = c_mods.rnd[t];
        const uint32_t m = c_mods.m[t];
#pragma unroll
        for (int b = 0; b < 4; b++) r[b] = acc_residue((int)v[b], rnd, m);
    } else {
#pragma unroll
        for (int b = 0; b < 4; b++) r[b] = acc_residue_any((int)v[b], t);
    }
    return pack_low_bytes(r[0], r[1], r[2], r[3]) ^ 0x80808080u;
}

// X [n_in][R] (uint64) -> XP [t][R][Kp] (int8), via 64 x 64 shared-memory transposes.  A block
// converts kXresTiles column tiles of one 64-input group: the next tile's rows are copied by
// cp.async (8-byte pieces; rows past n_in filled with zeros) while the current one is converted.
// Each thread writes four consecutive inputs' residues of one column as one 32-bit word, so a
// warp's store covers 64 contiguous bytes of each of two columns for every modulus.  F64 (every
// limb prime below 2^51): each residue from one FP64 and one integer multiply-add (balanced_f64),
// else in 32-bit integer arithmetic (mod_small).  T, the moduli, at compile time: a loop to the largest
// count under guards issued the guarded iterations too.
// What bounds it: HBM (768 inputs, 131,072 columns, 12 moduli: 2.0 GB a pass).  The input groups of a column
// tile are consecutive blocks, so the 64-byte pieces of a plane's row are written at about the same time and
// leave L2 as whole rows, and row i of a tile is rotated by i / 4 columns, so the 16 rows that a half-warp
// reads lie in different banks (unrotated, padded rows: four to a bank).  The two take 3.1 ms off 768 to 768
// ciphertexts at 13 limbs (29.1 in all), 0.11 off 100 to 70 at 7 limbs (1.71).
constexpr uint32_t kXresTiles = 2;
constexpr uint32_t kXresSmem = 2 * 64 * 64 * 8;

template <bool F64, uint32_t T>
__global__ void __launch_bounds__(256, 3) xres_kernel(const uint64_t *__restrict__ X, int8_t *__restrict__ XP,
                                                      uint32_t n_in, uint32_t Kp, uint64_t R, uint64_t r0,
                                                      uint64_t chunk) {
    extern __shared__ uint64_t xres_smem[];
    uint64_t(*tile)[64][64] = reinterpret_cast<uint64_t(*)[64][64]>(xres_smem);
    const uint32_t groups = Kp / 64, i0 = blockIdx.x % groups * 64;
    const uint32_t tx = threadIdx.x & 63, ty = threadIdx.x >> 6;  // 256 threads: 64 x 4
    const uint64_t rb0 = (uint64_t)(blockIdx.x / groups) * kXresTiles * 64;
    auto fetch = [&](uint32_t buf, uint64_t rb) {
        for (uint32_t i = ty; i < 64; i += 4) {
            const uint32_t ii = i0 + i;
            const uint64_t *src = X + (uint64_t)(ii < n_in ? ii : 0) * R + r0 + rb + tx;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(smem_u32(&tile[buf][i][(tx + (i >> 2)) & 63])),
                         "l"(src),
                         "r"(ii < n_in ? 8 : 0));
        }
        asm volatile("cp.async.commit_group;\n");
    };
    fetch(0, rb0);
    const uint32_t kq = threadIdx.x & 15, cg = threadIdx.x >> 4;  // inputs 4 kq .. 4 kq + 3, columns 4 cg .. 4 cg + 3
    for (uint32_t k = 0; k < kXresTiles; k++) {
        const uint32_t buf = k & 1;
        const uint64_t rb = rb0 + (uint64_t)k * 64;
        if (k + 1 < kXresTiles) {
            fetch(buf ^ 1, rb + 64);
            asm volatile("cp.async.wait_group 1;\n");
        } else {
            asm volatile("cp.async.wait_group 0;\n");
        }
        __syncthreads();
#pragma unroll
        for (uint32_t c = 0; c < 4; c++) {
            const uint32_t col = 4 * cg + c;
            uint64_t x[4];
#pragma unroll
            for (uint32_t j = 0; j < 4; j++) x[j] = tile[buf][4 * kq + j][(col + kq) & 63];
            int8_t *dst = XP + (rb + col) * Kp + i0 + 4 * kq;
            if constexpr (F64) {
                const double two52 = 4503599627370496.0;
                double xd[4];
                uint32_t xl[4];
#pragma unroll
                for (uint32_t j = 0; j < 4; j++) {  // exact: x < 2^51
                    xd[j] = __dsub_rn(__longlong_as_double((long long)(0x4330000000000000ull | x[j])), two52);
                    xl[j] = (uint32_t)x[j];
                }
#pragma unroll
                for (uint32_t t = 0; t < T; t++) {
                    *reinterpret_cast<uint32_t *>(dst + (uint64_t)t * chunk * Kp) =
                            pack_low_bytes(balanced_f64(xd[0], xl[0], t), balanced_f64(xd[1], xl[1], t),
                                           balanced_f64(xd[2], xl[2], t), balanced_f64(xd[3], xl[3], t));
                }
            } else {
                for (uint32_t t = 0; t < T; t++) {
                    uint32_t w = 0;
#pragma unroll
                    for (uint32_t j = 0; j < 4; j++)
                        w |= (uint32_t)(uint8_t)balanced(mod_small(x[j], t), c_mods.m[t]) << (8 * j);
                    *reinterpret_cast<uint32_t *>(dst + (uint64_t)t * chunk * Kp) = w;
                }
            }
        }
        __syncthreads();  // the buffer is refilled by the tile after next
    }
}

// W [n_in][n_out] (int64) -> WP [t][Np][Kp] (int8)
__global__ void wres_kernel(const int64_t *__restrict__ W, int8_t *__restrict__ WP, uint32_t n_in, uint32_t n_out,
                            uint32_t Kp, uint32_t Np, uint32_t T) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;  // input index (K)
    const uint32_t o = blockIdx.y;
    if (i >= Kp) return;
    int64_t w = (i < n_in && o < n_out) ? W[(uint64_t)i * n_out + o] : 0;
    for (uint32_t t = 0; t < T; t++) {
        int64_t m = c_mods.m[t];
        int64_t r = w % m;
        if (r < 0) r += m;
        WP[((uint64_t)t * Np + o) * Kp + i] = balanced((uint32_t)r, (uint32_t)m);
    }
}

// ---------------------------------------------------------------- tcgen05 GEMM

// K-major operand written by TMA with the 64-byte swizzle (rows of kKB = 64 bytes, 8-row groups
// 512 bytes apart); the MMA over K bytes [32 k, 32 k + 32) starts 32 k bytes into the atom
__device__ __forceinline__ uint64_t smem_desc_sw64(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFF);
    d |= (uint64_t)1 << 16;           // leading byte offset: unused within one swizzle atom
    d |= (uint64_t)(512 >> 4) << 32;  // stride byte offset: 8 rows x 64 bytes
    d |= (uint64_t)1 << 46;           // descriptor version for sm_100
    d |= (uint64_t)4 << 61;           // layout: SWIZZLE_64B
    return d;
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src));
}

// grid: (Np / 128, R_chunk / 256, T); one modulus per blockIdx.z.  D[o][r] = W[o] . X[r]: the
// weights are A (128 outputs, TMEM lanes), the X residues B (256 columns, TMEM columns), so an
// epilogue thread holds 32 consecutive columns of one output and writes them as two 16-byte
// stores.  The output tiles are the fastest grid dimension: the CTAs that share an X tile
// run together and read it from HBM once (then from L2).  Two CTAs per SM (2 x 97 KB shared
// memory, 2 x 256 TMEM columns).
//
// Warp-specialised: warps 0-3 fill a kStages-deep ring with cp.async (each producer thread
// waits for its own copies of the previous stage, fences them into the async proxy and
// arrives on that stage's `full` barrier); one thread of warp 4 issues the MMAs of a stage
// once it is full and frees it through tcgen05.commit on its `empty` barrier; after the
// last commit (`done`) all eight warps read the accumulators back.  No block-wide barrier
// inside the K loop; every wait is bounded (a timeout sets *err and skips the stores).
__global__ void __launch_bounds__(kThreads, 2) mma_kernel(const int8_t *__restrict__ XP, const int8_t *__restrict__ WP,
                                                          uint8_t *__restrict__ RES, uint32_t Kp, uint32_t Np,
                                                          uint32_t n_out, uint64_t chunk, int *__restrict__ err,
                                                          int acc_small, int limit) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[kStages], empty[kStages], done;
    __shared__ uint32_t tmem_base;
    __shared__ int failed;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t t = blockIdx.z;
    const uint64_t rbase = (uint64_t)blockIdx.y * kBN;
    const uint32_t obase = blockIdx.x * kBM;
    const int8_t *A = WP + ((uint64_t)t * Np + obase) * Kp;     // [128][Kp]
    const int8_t *B = XP + ((uint64_t)t * chunk + rbase) * Kp;  // [256][Kp]
    uint8_t *sA = smem, *sB = smem + kStages * kStageA;
    constexpr uint32_t kProducers = 128;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_base)),
                     "r"(kBN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    if (tid == 0) {
        for (int s = 0; s < kStages; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(&full[s])), "r"(kProducers));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&empty[s])));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&done)));
        asm volatile("fence.mbarrier_init.release.cluster;\n");
        failed = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    const uint32_t tmem = tmem_base;
    const uint32_t nkb = Kp / kKB;
    // instruction descriptor: s32 accumulate, A and B signed int8, both K-major, N = 256, M = 128
    const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((kBN >> 3) << 17) | ((kBM >> 4) << 24);

    if (tid < kProducers) {
        bool ok = true;
        for (uint32_t kb = 0; kb < nkb; kb++) {
            const uint32_t s = kb % kStages;
            if (ok && kb >= (uint32_t)kStages && !mbar_wait(smem_u32(&empty[s]), ((kb / kStages) - 1) & 1, limit)) ok = false;
            const uint32_t a_dst = smem_u32(sA + s * kStageA), b_dst = smem_u32(sB + s * kStageB);
            const uint64_t koff = (uint64_t)kb * kKB;
            if (ok) {
                for (uint32_t c = tid; c < kBM * (kKB / 16); c += kProducers) {
                    const uint32_t row = c / (kKB / 16), kc = c % (kKB / 16);
                    cp_async16(a_dst + core_off(row, kc), A + (uint64_t)row * Kp + koff + kc * 16);
                }
                for (uint32_t c = tid; c < kBN * (kKB / 16); c += kProducers) {
                    const uint32_t row = c / (kKB / 16), kc = c % (kKB / 16);
                    cp_async16(b_dst + core_off(row, kc), B + (uint64_t)row * Kp + koff + kc * 16);
                }
            }
            asm volatile("cp.async.commit_group;\n");
            if (kb >= 1) {  // this thread's copies of stage kb - 1 have landed
                asm volatile("cp.async.wait_group 1;\n");
                asm volatile("fence.proxy.async.shared::cta;\n");
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(&full[(kb - 1) % kStages])));
            }
        }
        asm volatile("cp.async.wait_group 0;\n");
        asm volatile("fence.proxy.async.shared::cta;\n");
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(&full[(nkb - 1) % kStages])));
        if (!ok) failed = 1;
    } else if (tid == kProducers) {
        bool ok = true;
        for (uint32_t kb = 0; kb < nkb; kb++) {
            const uint32_t s = kb % kStages;
            if (ok && !mbar_wait(smem_u32(&full[s]), (kb / kStages) & 1, limit)) ok = false;
            asm volatile("tcgen05.fence::after_thread_sync;\n");
            if (ok) {
                const uint32_t a0 = smem_u32(sA + s * kStageA), b0 = smem_u32(sB + s * kStageB);
#pragma unroll
                for (uint32_t k = 0; k < kKB / 32; k++) {
                    uint64_t ad = smem_desc(a0 + k * 256), bd = smem_desc(b0 + k * 256);
                    uint32_t acc = (kb | k) ? 1u : 0u;
                    asm volatile(
                        "{\n\t.reg .pred p;\n\t"
                        "setp.ne.b32 p, %4, 0;\n\t"
                        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
                        "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
                }
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                smem_u32(&empty[s])));
        }
        // completes once every MMA above has
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
            smem_u32(&done)));
        if (!ok) failed = 1;
    }
    // the idle warps wait here instead of spinning beside the producers and the MMA thread
    __syncthreads();  // also publishes `failed` from the producer and MMA roles
    const bool landed = __all_sync(0xffffffffu, mbar_wait(smem_u32(&done), 0, limit));
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    if (!landed || failed) {
        if (lane == 0) atomicExch(err, 1);
        if (!landed) mbar_wait(smem_u32(&done), 0);  // once more, for the MMAs in flight: the TMEM is freed next
    } else {
        // epilogue: warp w reads TMEM lanes 32 (w % 4) .. + 31 (outputs); warpgroup w / 4 takes one
        // half of the 256 X columns, 32 at a time
        const uint32_t quarter = warp & 3, half = warp >> 2;
        const uint32_t o = obase + quarter * 32 + lane;
        for (uint32_t c0 = half * (kBN / 2); c0 < (half + 1) * (kBN / 2); c0 += 32) {
            uint32_t v[32];
            const uint32_t taddr = tmem + ((quarter * 32) << 16) + c0;
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
                : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                  "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                  "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]),
                  "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]),
                  "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                : "r"(taddr));
            asm volatile("tcgen05.wait::ld.sync.aligned;\n");
            if (o < n_out) {
                uint32_t pk[8];
#pragma unroll
                for (int j = 0; j < 8; j++) pk[j] = acc_bytes(v + 4 * j, t, acc_small);
                uint4 *dst = reinterpret_cast<uint4 *>(RES + ((uint64_t)t * n_out + o) * chunk + rbase + c0);
                dst[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                dst[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kBN));
}

// ---------------------------------------------------------------- persistent GEMM
// For K <= kResKp the 256-column X tile of one modulus stays resident in shared memory (Kp / 64
// blocks of 16 KB in the MMA's core-matrix layout) while the CTA runs every output tile of it:
// the weight tiles (A, 128 outputs x 64 K bytes) stream through a kAStages ring, and the
// accumulators alternate between two 256-column TMEM buffers so that the epilogue of one output
// tile overlaps the MMAs of the next.  One CTA per SM (all 512 TMEM columns), persistent over
// the (modulus, column tile) pairs.  Roles: warps 0-3 copy (cp.async; the X tile together, then
// the A stages, warp w filling ring slot w and arriving on its barrier once its copies land, the
// next X tile prefetched into L2 meanwhile), one thread of warp 4
// issues the MMAs, warps 5-12 read the accumulators back (two warps per 32-lane quarter, one
// per half of the columns).  Every wait is bounded; a role whose wait runs out leaves its loops, and the
// others, whose polls look at `failed`, leave theirs.  The loads and MMAs in flight are then waited for (again
// with a bound) before the CTA frees its TMEM and ends, and the call reports the failure through *err.
constexpr uint32_t kResKp = 768;
constexpr int kAStages = 4;  // one ring slot per producer warp
constexpr uint32_t kXBlock = kBN * kKB;  // 16 KB
constexpr uint32_t kXTiles = 6;          // most X tiles held at a time
constexpr uint32_t kSmemP = (kResKp / kKB) * kXBlock + kAStages * kStageA + 1024;
constexpr uint32_t kEpiWarp0 = 5;
constexpr uint32_t kThreadsP = (kEpiWarp0 + 8) * 32;

// a role's wait: false, with *failed set, once it or another role's has run out
__device__ __forceinline__ bool role_wait(uint32_t bar, uint32_t parity, int limit, volatile int *failed) {
    for (int it = 0; it < limit; it++) {
        if (mbar_try(bar, parity)) return true;
        if (*failed) return false;
    }
    *failed = 1;
    return false;
}

// TMA_A: both operands come by TMA (one thread issues the X tile's and the weight stages' loads,
// 64-byte swizzle, completion on their mbarriers) instead of the producer warps' cp.async.  LIMITED: `limit` polls a
// wait instead of kSpinLimit (a run-time bound of every wait: 1.33 ms for 1.26 a pass of 768 x 768)
template <bool TMA_A, bool LIMITED>
__global__ void __launch_bounds__(kThreadsP, 1) mma_persistent_kernel(const int8_t *__restrict__ XP,
                                                                      const int8_t *__restrict__ WP,
                                                                      uint8_t *__restrict__ RES, uint32_t Kp,
                                                                      uint32_t Np, uint32_t n_out, uint64_t chunk,
                                                                      uint32_t T, int *__restrict__ err, int acc_small,
                                                                      int limit,
                                                                      const __grid_constant__ CUtensorMap tmA,
                                                                      const __grid_constant__ CUtensorMap tmX) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);  // swizzle atoms need 1 KB alignment
    __shared__ __align__(8) uint64_t full[kAStages], empty[kAStages], x_full[kXTiles], x_empty[kXTiles], acc_full[2],
        acc_empty[2], drained;
    __shared__ uint32_t tmem_base;
    __shared__ int failed;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint8_t *sX = smem, *sA = smem + (kResKp / kKB) * kXBlock;
    const uint32_t nkb = Kp / kKB, n_ot = Np / kBM;
    const uint64_t n_ct = chunk / kBN, n_tiles = (uint64_t)T * n_ct;
    // X tiles held: tile i of this CTA in slot i % ns.  At K = 768 one fits; small K (where a tile's load, MMAs and
    // epilogue came one after another: 4.7 us per tile of 128 inputs) has the next ones loaded ahead.
    const uint32_t ns = min(kXTiles, kResKp / Kp);
    constexpr uint32_t kProducers = 128, kEpi = 256;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_base)),
                     "r"(2 * kBN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    if (tid == 0) {
        for (int s = 0; s < kAStages; s++) {
            // the TMA issuer's expect-tx arrival, or the 32 threads of the slot's producer warp
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(&full[s])), "r"(TMA_A ? 1 : 32));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&empty[s])));
        }
        for (uint32_t x = 0; x < kXTiles; x++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(&x_full[x])),
                         "r"(TMA_A ? 1 : kProducers));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&x_empty[x])));
        }
        for (int b = 0; b < 2; b++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&acc_full[b])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(&acc_empty[b])), "r"(kEpi));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&drained)));
        asm volatile("fence.mbarrier_init.release.cluster;\n");
        failed = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    const uint32_t tmem = tmem_base;
    const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((kBN >> 3) << 17) | ((kBM >> 4) << 24);
    auto wait = [&](uint64_t *bar, uint32_t parity) { return role_wait(smem_u32(bar), parity, LIMITED ? limit : kSpinLimit, &failed); };
    auto arrive = [](uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar)); };

    if (tid < kProducers && !(TMA_A && warp > 0)) {
        // cp.async: producer warp w fills ring slot w (A stages w, w + 4, ...): each warp waits for
        // its own copies only, so four stages are in flight; all four copy the X tile together.
        // TMA: thread 0 issues every load (the X tile as Kp / 64 boxes of 256 rows, then the A
        // stages), its warp prefetches the next X tile into L2
        bool ok = true;
        uint32_t g = 0;   // A stages so far (ring position)
        uint32_t ti = 0;  // column tiles of this CTA so far
        uint32_t xi = 0;  // X tiles asked for so far (TMA)
        const uint32_t kx16 = Kp / 16;
        // every MMA of the slot's previous tile must have read it
        auto x_free = [&](uint32_t i) { return i < ns || wait(&x_empty[i % ns], (i / ns - 1) & 1); };
        for (uint64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ti++) {
            const uint32_t t = (uint32_t)(tile / n_ct);
            const uint64_t rbase = (tile % n_ct) * kBN;
            if constexpr (TMA_A) {
                // ahead of this tile's weights: the X tiles whose slots' last readers came two tiles ago
                if (tid == 0)
                    for (; ok && xi <= (ns > 1 ? ti + ns - 2 : ti); xi++) {
                        const uint64_t xt = blockIdx.x + (uint64_t)xi * gridDim.x;
                        if (xt >= n_tiles) break;
                        if (!x_free(xi)) {
                            ok = false;
                            break;
                        }
                        const uint32_t bar = smem_u32(&x_full[xi % ns]);
                        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar),
                                     "r"(kBN * Kp));
                        for (uint32_t kb = 0; kb < nkb; kb++)  // x = kb * 64 bytes: 16-byte aligned
                            asm volatile(
                                "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
                                "[%0], [%1, {%2, %3}], [%4];\n" ::"r"(smem_u32(sX + (xi % ns * nkb + kb) * kXBlock)),
                                "l"(reinterpret_cast<uint64_t>(&tmX)), "r"((int)(kb * kKB)),
                                "r"((int)((xt / n_ct) * chunk + (xt % n_ct) * kBN)), "r"(bar)
                                : "memory");
                    }
                ok = __shfl_sync(0xffffffffu, ok, 0);  // thread 0's, also from the tile before
                if (!ok) break;
            } else {
                if (!x_free(ti)) break;
                const int8_t *B = XP + ((uint64_t)t * chunk + rbase) * Kp;
                for (uint32_t c = tid; c < kBN * kx16; c += kProducers) {
                    const uint32_t row = c / kx16, k16 = c % kx16;
                    cp_async16(smem_u32(sX + (ti % ns * nkb + (k16 >> 2)) * kXBlock) + core_off(row, k16 & 3),
                               B + (uint64_t)row * Kp + k16 * 16);
                }
                asm volatile("cp.async.commit_group;\n");
                asm volatile("cp.async.wait_group 0;\n");
                asm volatile("fence.proxy.async.shared::cta;\n");
                arrive(smem_u32(&x_full[ti % ns]));
            }
            // the next column tile's X into L2 while this one's MMAs run
            const uint64_t next = tile + gridDim.x;
            if (next < n_tiles) {
                const int8_t *Bn = XP + ((uint64_t)(next / n_ct) * chunk + (next % n_ct) * kBN) * Kp;
                const uint32_t nthr = TMA_A ? 32 : kProducers;
                for (uint32_t off = tid * 128; off < kBN * Kp; off += nthr * 128)
                    asm volatile("prefetch.global.L2 [%0];\n" ::"l"(Bn + off));
            }
            for (uint32_t o = 0; ok && o < n_ot; o++) {
                const int8_t *A = WP + ((uint64_t)t * Np + o * kBM) * Kp;
                for (uint32_t kb = 0; kb < nkb; kb++, g++) {
                    const uint32_t s = (uint32_t)(g % kAStages);
                    if (TMA_A ? tid != 0 : s != warp) continue;
                    if (g >= (uint32_t)kAStages && !wait(&empty[s], (uint32_t)((g / kAStages) - 1) & 1)) {
                        ok = false;
                        break;
                    }
                    const uint32_t bar = smem_u32(&full[s]);
                    if constexpr (TMA_A) {
                        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar),
                                     "r"(kStageA));
                        // x = kb * 64 bytes: 16-byte aligned as a tiled TMA load requires
                        asm volatile(
                            "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
                            "[%0], [%1, {%2, %3}], [%4];\n" ::"r"(smem_u32(sA + s * kStageA)),
                            "l"(reinterpret_cast<uint64_t>(&tmA)), "r"((int)(kb * kKB)),
                            "r"((int)(t * Np + o * kBM)), "r"(bar)
                            : "memory");
                    } else {
                        for (uint32_t c = lane; c < kBM * (kKB / 16); c += 32) {
                            const uint32_t row = c / (kKB / 16), kc = c % (kKB / 16);
                            cp_async16(smem_u32(sA + s * kStageA) + core_off(row, kc),
                                       A + (uint64_t)row * Kp + (uint64_t)kb * kKB + kc * 16);
                        }
                        asm volatile("cp.async.commit_group;\n");
                        asm volatile("cp.async.wait_group 0;\n");
                        asm volatile("fence.proxy.async.shared::cta;\n");
                        arrive(bar);
                    }
                }
            }
            if (!TMA_A && !ok) break;
        }
        if (TMA_A && tid == 0) {  // every load asked for has landed (normally long ago) before the CTA can end
            for (uint32_t s = 0; s < (uint32_t)kAStages; s++)
                if (g > s) mbar_wait(smem_u32(&full[s]), ((g - 1 - s) / kAStages) & 1);
            for (uint32_t x = 0; x < ns; x++)
                if (xi > x) mbar_wait(smem_u32(&x_full[x]), ((xi - 1 - x) / ns) & 1);
        }
    } else if (tid == kProducers) {
        bool ok = true;
        uint32_t g = 0, ti = 0, ai = 0;  // A stages, column tiles, accumulator tiles
        for (uint64_t tile = blockIdx.x; ok && tile < n_tiles; tile += gridDim.x, ti++) {
            const uint32_t xs = ti % ns;
            ok = wait(&x_full[xs], (ti / ns) & 1);
            asm volatile("tcgen05.fence::after_thread_sync;\n");
            for (uint32_t o = 0; ok && o < n_ot; o++, ai++) {
                const uint32_t buf = ai & 1;
                if (ai >= 2 && !wait(&acc_empty[buf], ((ai >> 1) - 1) & 1)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n");
                for (uint32_t kb = 0; kb < nkb; kb++, g++) {
                    const uint32_t s = (uint32_t)(g % kAStages);
                    if (!wait(&full[s], (uint32_t)(g / kAStages) & 1)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;\n");
                    const uint32_t a0 = smem_u32(sA + s * kStageA), b0 = smem_u32(sX + (xs * nkb + kb) * kXBlock);
#pragma unroll
                    for (uint32_t k = 0; k < kKB / 32; k++) {
                        const uint64_t ad = TMA_A ? smem_desc_sw64(a0 + k * 32) : smem_desc(a0 + k * 256);
                        const uint64_t bd = TMA_A ? smem_desc_sw64(b0 + k * 32) : smem_desc(b0 + k * 256);
                        const uint32_t accum = (kb | k) ? 1u : 0u;
                        asm volatile(
                            "{\n\t.reg .pred p;\n\t"
                            "setp.ne.b32 p, %4, 0;\n\t"
                            "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem + buf * kBN),
                            "l"(ad), "l"(bd), "r"(idesc), "r"(accum));
                    }
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                        smem_u32(&empty[s])));
                }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                    smem_u32(&acc_full[buf])));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                smem_u32(&x_empty[xs])));
        }
    } else if (warp >= kEpiWarp0) {
        bool ok = true;
        const uint32_t quarter = warp & 3, half = (warp - kEpiWarp0) >> 2;
        uint32_t ai = 0;
        for (uint64_t tile = blockIdx.x; ok && tile < n_tiles; tile += gridDim.x) {
            const uint32_t t = (uint32_t)(tile / n_ct);
            const uint64_t rbase = (tile % n_ct) * kBN;
            for (uint32_t o = 0; o < n_ot; o++, ai++) {
                const uint32_t buf = ai & 1;
                ok = __all_sync(0xffffffffu, wait(&acc_full[buf], (ai >> 1) & 1));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n");
                const uint32_t out = o * kBM + quarter * 32 + lane;
                for (uint32_t c0 = half * (kBN / 2); c0 < (half + 1) * (kBN / 2); c0 += 32) {
                    uint32_t v[32];
                    const uint32_t taddr = tmem + ((quarter * 32) << 16) + buf * kBN + c0;
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
                        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
                          "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
                          "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]),
                          "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]),
                          "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                        : "r"(taddr));
                    asm volatile("tcgen05.wait::ld.sync.aligned;\n");
                    if (out < n_out) {
                        uint32_t pk[8];
#pragma unroll
                        for (int j = 0; j < 8; j++) pk[j] = acc_bytes(v + 4 * j, t, acc_small);
                        uint4 *dst = reinterpret_cast<uint4 *>(RES + ((uint64_t)t * n_out + out) * chunk + rbase + c0);
                        dst[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                        dst[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;\n");
                arrive(smem_u32(&acc_empty[buf]));
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    if (failed) {
        if (tid == 0) atomicExch(err, 1);
        if (tid == kProducers) {  // the MMAs in flight
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                smem_u32(&drained)));
            mbar_wait(smem_u32(&drained), 0);
        }
        asm volatile("tcgen05.fence::before_thread_sync;\n");
        __syncthreads();
    }
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(2 * kBN));
}

// ---------------------------------------------------------------- CRT fold
struct CrtLimb {
    uint64_t c[kMaxMods];  // c_t mod q_l
    uint64_t Mneg;         // q_l - (M mod q_l), below q_l
    uint64_t base;         // 128 T M - 128 sum_t c_t mod q_l
};

// Fraction bits of the fixed-point CRT fractions F_t = round(2^19 [(M/m_t)^-1]_{m_t} / m_t).  The planes hold
// u_t = r_t + 128 with |r_t| <= 127, so v = round(sum_t r_t frac_t) is found as v + 128 T from
// sum_t u_t F_t + vbase, vbase = 128 T 2^19 - 128 sum_t F_t + 2^18: non-negative and below 2^32 for T <= 20.
// The rounding error T 128 2^-20 < 0.003 keeps v exact (M > 2.02 |S| leaves the true sum within 0.495 of
// an integer).
constexpr uint32_t kCrtFracBits = 19;

// workspace bytes before the residue planes: the error flag, then the CRT tables for every
// moduli count in use (at most kMaxMods counts of up to 64 limbs)
constexpr size_t kCrtTabBytes = 256 + sizeof(CrtLimb) * 64 * kMaxMods;

// One thread folds 4 consecutive columns r of one output (4-byte residue loads, two 16-byte
// stores).  The host sizes the block so that its 4 blockDim.x columns lie in one limb: the limb's
// constants are staged in shared memory once per block.  The sums over t, exact:
//   lo = sum u_t (c_t mod 2^32),  hi = sum u_t (c_t >> 32),  v = sum u_t F_t  (32-bit fixed point),
// then S = sum_t r_t c_t - v M = base + lo + hi 2^32 + (v + 128 T) (q - M mod q) mod q, base taking the
// offsets back, one Barrett reduction (the sum is below 20 255 2^61 + 2^13 2^61 < 2^75).
// HI32: the host has checked that (T 255 + 1) max(q >> 32) < 2^32 (so q < 2^56) and every q >= 2^40.  Then
// hi fits 32 bits and one FP64 quotient replaces Barrett's two 64 x 64-bit high products, and the sums are
// taken byte by byte: four moduli's residues of a column (a 4 x 4 byte transpose) times the same four moduli's
// bytes of c_t (seven) and F_t (three) are ten four-way byte products, 30 a column for 12 moduli in place of
// 12 wide and 24 plain multiply-adds and 12 byte extracts.  They take 0.7 ms off
// 768 to 768 ciphertexts at 13 limbs, 0.04 off 100 to 70 at 7 limbs (alternated runs).  The residue words (one per modulus,
// read once: streaming loads) are requested before the fold.  T at compile time, as in xres_kernel (232
// instructions a column were issued for 12 moduli under guards up to 20: 0.77 ms a pass of 768 x 131,072).
template <bool HI32, uint32_t T>
__global__ void __launch_bounds__(256) crt_kernel(const uint8_t *__restrict__ RES, uint64_t *__restrict__ Y,
                                                  const CrtLimb *__restrict__ tab, uint32_t n_out, uint64_t chunk,
                                                  uint64_t r0, uint64_t R, uint32_t L, uint32_t log_n,
                                                  const PrimeConst *__restrict__ pc) {
    constexpr uint32_t G = (T + 3) / 4;  // groups of four moduli
    __shared__ uint32_t s_lo[kMaxMods], s_hi[kMaxMods], s_f[kMaxMods];
    __shared__ __align__(16) uint32_t s_k[G][12];
    const uint64_t rb = (uint64_t)blockIdx.x * blockDim.x * 4;
    const uint32_t o = blockIdx.y;
    const uint32_t row = (uint32_t)((r0 + rb) >> log_n);  // h L + limb, below 2 L
    const uint32_t limb = row >= L ? row - L : row;
    if constexpr (HI32) {
        for (uint32_t i = threadIdx.x; i < G * 12; i += blockDim.x) {
            const uint32_t g = i / 12, b = i % 12;
            uint32_t w = 0;
#pragma unroll
            for (uint32_t j = 0; j < 4; j++) {
                const uint32_t t = 4 * g + j;
                if (t < T && b < 10) {
                    const uint32_t byte = b < 7 ? (uint32_t)(tab[limb].c[t] >> (8 * b)) : c_mods.fracq[T][t] >> (8 * (b - 7));
                    w |= (byte & 0xFF) << (8 * j);
                }
            }
            s_k[g][b] = w;
        }
    } else if (threadIdx.x < T) {
        const uint32_t t = threadIdx.x;
        const uint64_t c = tab[limb].c[t];
        s_lo[t] = (uint32_t)c;
        s_hi[t] = (uint32_t)(c >> 32);
        s_f[t] = c_mods.fracq[T][t];
    }
    __syncthreads();
    const uint64_t r = rb + (uint64_t)threadIdx.x * 4;
    if (r >= chunk) return;
    const uint64_t rg = r0 + r;
    const PrimeConst p = pc[limb];
    const uint64_t Mneg = tab[limb].Mneg;
    const double k32 = __dmul_rn(4294967296.0, p.qinv);
    uint32_t res[4 * G];  // requested before the fold
#pragma unroll
    for (uint32_t t = 0; t < T; t++)
        res[t] = __ldcs(reinterpret_cast<const uint32_t *>(RES + ((uint64_t)t * n_out + o) * chunk + r));
#pragma unroll
    for (uint32_t t = T; t < 4 * G; t++) res[t] = 0;
    const uint64_t base = tab[limb].base;
    const uint32_t vbase = c_mods.vbase[T];
    uint64_t y[4];
    if constexpr (HI32) {
        uint32_t d[4][10];
#pragma unroll
        for (int e = 0; e < 4; e++) {
#pragma unroll
            for (int b = 0; b < 10; b++) d[e][b] = 0;
            d[e][0] = (uint32_t)base & 0xFFFF;
            d[e][2] = (uint32_t)base >> 16;
            d[e][4] = (uint32_t)(base >> 32);
            d[e][7] = vbase & 0xFFFF;
            d[e][9] = vbase >> 16;
        }
#pragma unroll
        for (uint32_t g = 0; g < G; g++) {
            const uint32_t *w = res + 4 * g;  // four moduli of four columns -> four columns of four moduli
            const uint32_t a0 = __byte_perm(w[0], w[1], 0x5140), a1 = __byte_perm(w[2], w[3], 0x5140);
            const uint32_t a2 = __byte_perm(w[0], w[1], 0x7362), a3 = __byte_perm(w[2], w[3], 0x7362);
            const uint32_t u[4] = {__byte_perm(a0, a1, 0x5410), __byte_perm(a0, a1, 0x7632),
                                   __byte_perm(a2, a3, 0x5410), __byte_perm(a2, a3, 0x7632)};
            uint32_t k[12];
#pragma unroll
            for (int b = 0; b < 12; b += 4) {
                const uint4 x = *reinterpret_cast<const uint4 *>(&s_k[g][b]);
                k[b] = x.x, k[b + 1] = x.y, k[b + 2] = x.z, k[b + 3] = x.w;
            }
#pragma unroll
            for (int e = 0; e < 4; e++)
#pragma unroll
                for (int b = 0; b < 10; b++) d[e][b] = __dp4a(u[e], k[b], d[e][b]);
        }
#pragma unroll
        for (int e = 0; e < 4; e++) {
            // S = H 2^32 + l with H < 2^34: Q = round(H 2^32 / q) from the FP64 pipe, S - Q q is within
            // q/2 + 2^32 of zero (q >= 2^40)
            const uint32_t w = (d[e][7] + (d[e][8] << 8) + (d[e][9] << 16)) >> kCrtFracBits;
            const uint64_t l = (d[e][0] + (d[e][1] << 8)) + ((uint64_t)(d[e][2] + (d[e][3] << 8)) << 16) +
                               (uint64_t)w * (uint32_t)Mneg;
            const uint64_t H = (uint64_t)w * (uint32_t)(Mneg >> 32) +
                               (d[e][4] + (d[e][5] << 8) + (d[e][6] << 16)) + (l >> 32);
            const double hd = __dsub_rn(as_dbl(0x4330000000000000ull | H), kTwo52);
            const uint32_t Q = (uint32_t)as_bits(__fma_rn(hd, k32, kTwo52));
            const uint64_t x = ((H << 32) | (uint32_t)l) - Q * p.q;
            y[e] = x + ((uint64_t)((int64_t)x >> 63) & p.q);
        }
    } else {
        uint64_t lo[4], hi[4];
        uint32_t v[4];
#pragma unroll
        for (int e = 0; e < 4; e++) lo[e] = (uint32_t)base, hi[e] = base >> 32, v[e] = vbase;
#pragma unroll
        for (uint32_t t = 0; t < T; t++) {
            const uint32_t cl = s_lo[t], ch = s_hi[t], f = s_f[t];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const uint32_t rt = (res[t] >> (8 * e)) & 0xFF;
                lo[e] += (uint64_t)rt * cl;
                hi[e] += (uint64_t)rt * ch;
                v[e] += rt * f;
            }
        }
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const uint64_t h = hi[e], w = v[e] >> kCrtFracBits;
            const uint64_t plo = lo[e] + (h << 32);
            u128 pos = {plo, (h >> 32) + (plo < lo[e] ? 1ull : 0ull)};
            mac(pos, w, Mneg);
            y[e] = barrett(pos, p);
        }
    }
    ulonglong2 *out = reinterpret_cast<ulonglong2 *>(Y + (uint64_t)o * R + rg);
    out[0] = make_ulonglong2(y[0], y[1]);
    out[1] = make_ulonglong2(y[2], y[3]);
}

}  // namespace

// ------------------------------------------------------------------ host side

namespace {

struct Plan {
    ModTab mods;
    uint32_t T_min = 0, T_max = 0;   // the moduli counts the limbs need
    std::vector<uint32_t> limb_T;    // per limb
    std::vector<CrtLimb> limbs;      // [T - T_min][L]: the CRT constants for each count in use
    bool hi32 = false;               // the CRT's high sums in 32 bits (crt_kernel)
};

// The moduli count of each limb: |S| = |sum_i x_i w_io| <= (q_l - 1) max_o sum_i |w_io| = B_l, and
// the CRT with the fixed-point v (error below 0.005) is exact while M > 2 B_l / (1 - 0.01); the
// product of the first T candidates must exceed that (log2 M >= log2 B_l + 1.05).
Plan make_plan(const Context &c, uint32_t L, uint64_t max_l1) {
    static const uint32_t cand[kMaxMods] = {251, 241, 239, 233, 229, 227, 223, 211, 199, 197,
                                            193, 191, 181, 179, 173, 167, 163, 157, 151, 149};
    Plan p{};
    p.limb_T.resize(L);
    p.T_min = kMaxMods;
    uint64_t max_hi = 0, min_q = ~0ull;
    for (uint32_t l = 0; l < L; l++) {
        const uint64_t q = c.primes[l];
        const double need = std::log2((double)(q - 1)) + std::log2((double)std::max<uint64_t>(max_l1, 1)) + 1.05;
        double have = 0;
        uint32_t T = 0;
        while (have < need) {
            if (T >= (uint32_t)kMaxMods) throw std::invalid_argument("ct-pt matmul: weights or inputs too large");
            have += std::log2((double)cand[T]);
            T++;
        }
        p.limb_T[l] = T;
        p.T_min = std::min(p.T_min, T);
        p.T_max = std::max(p.T_max, T);
        max_hi = std::max(max_hi, (q - 1) >> 32);
        min_q = std::min(min_q, q);
    }
    p.hi32 = ((uint64_t)p.T_max * 255 + 1) * max_hi < (1ull << 32) && min_q >= (1ull << 40);
    for (uint32_t t = 0; t < (uint32_t)kMaxMods; t++) {
        const uint32_t m = cand[t];
        p.mods.m[t] = m;
        p.mods.c24[t] = (1u << 20) % m;
        p.mods.c48[t] = (uint32_t)((uint64_t)p.mods.c24[t] * p.mods.c24[t] % m);
        p.mods.magic[t] = (uint32_t)(((1ull << 32) + m - 1) / m);
        p.mods.inv[t] = 1.0 / m;
        p.mods.rnd[t] = (int)(((1ull << 32) + m / 2) / m);
    }
    // CRT fractions [(M/m_t)^-1 mod m_t] / m_t in fixed point, for every modulus count
    for (uint32_t n = 1; n <= (uint32_t)kMaxMods; n++)
        for (uint32_t t = 0; t < n; t++) {
            const uint32_t m = cand[t];
            uint32_t Mt_mod_m = 1;
            for (uint32_t u = 0; u < n; u++)
                if (u != t) Mt_mod_m = (uint32_t)((uint64_t)Mt_mod_m * (cand[u] % m) % m);
            const uint32_t inv = (uint32_t)host::powmod(Mt_mod_m, m - 2, m);  // m prime
            p.mods.fracq[n][t] = (uint32_t)((((uint64_t)inv << kCrtFracBits) + m / 2) / m);
        }
    for (uint32_t n = 1; n <= (uint32_t)kMaxMods; n++) {
        int64_t v = ((int64_t)(128 * n) << kCrtFracBits) + (1 << (kCrtFracBits - 1));
        for (uint32_t t = 0; t < n; t++) v -= 128 * (int64_t)p.mods.fracq[n][t];
        p.mods.vbase[n] = (uint32_t)v;
    }
    // CRT constants for each count T in use: c_t = (M/m_t) * [(M/m_t)^-1 mod m_t] mod q_l
    p.limbs.resize((size_t)(p.T_max - p.T_min + 1) * L);
    for (uint32_t T = p.T_min; T <= p.T_max; T++)
        for (uint32_t l = 0; l < L; l++) {
            CrtLimb &cl = p.limbs[(size_t)(T - p.T_min) * L + l];
            uint64_t q = c.primes[l], M = 1;
            for (uint32_t u = 0; u < T; u++) M = host::mulmod(M, cand[u], q);
            cl.Mneg = (q - M) % q;
            for (uint32_t t = 0; t < T; t++) {
                uint32_t m = cand[t], Mt_mod_m = 1;
                uint64_t Mt = 1;
                for (uint32_t u = 0; u < T; u++)
                    if (u != t) {
                        Mt = host::mulmod(Mt, cand[u], q);
                        Mt_mod_m = (uint32_t)((uint64_t)Mt_mod_m * (cand[u] % m) % m);
                    }
                uint32_t inv = (uint32_t)host::powmod(Mt_mod_m, m - 2, m);
                cl.c[t] = host::mulmod(Mt, inv, q);
                cl.base = (cl.base + q - host::mulmod(128, cl.c[t], q)) % q;
            }
            cl.base = (cl.base + host::mulmod(128 * T, M, q)) % q;
        }
    return p;
}

}  // namespace

// Residue planes [rows][Kp] (the weights' or X's) as a 2D tensor map for TMA: 64-byte K boxes of
// box_rows rows with the 64-byte swizzle.  False when the driver's encoder is unavailable or
// refuses, or when the environment sets SHMOAI_CTPT_TMA=0 (then the producer warps copy the
// operand tiles with cp.async).
bool operand_tensor_map(CUtensorMap *map, const int8_t *P, uint32_t Kp, uint64_t rows, uint32_t box_rows) {
    static PFN_cuTensorMapEncodeTiled encode = [] {
        const char *off = std::getenv("SHMOAI_CTPT_TMA");
        if (off && off[0] == '0') return (PFN_cuTensorMapEncodeTiled) nullptr;
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            fn = nullptr;
        cudaGetLastError();
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled>(fn);
    }();
    if (!encode) return false;
    const cuuint64_t dims[2] = {Kp, rows}, strides[1] = {Kp};
    const cuuint32_t box[2] = {kKB, box_rows}, estr[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<int8_t *>(P), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// columns of X processed per pass (bounds the residue workspaces); the environment variable
// SHMOAI_CTPT_CHUNK (a multiple of 256) replaces the default, read once per process
constexpr uint64_t kChunkCols = 131072;

static uint64_t chunk_cols() {
    static const uint64_t v = [] {
        const char *s = std::getenv("SHMOAI_CTPT_CHUNK");
        const uint64_t c = s ? std::strtoull(s, nullptr, 10) : 0;
        return (c >= kBN && c % kBN == 0) ? c : kChunkCols;
    }();
    return v;
}

size_t ctpt_tc_ws_bytes(const Context &c, uint32_t n_in, uint32_t n_out, uint32_t L) {
    const uint64_t R = 2ull * L * c.n;
    const uint64_t chunk = std::min<uint64_t>(R, chunk_cols());
    const uint32_t Kp = (n_in + kKB - 1) / kKB * kKB, Np = (n_out + kBM - 1) / kBM * kBM;
    return (size_t)kMaxMods * (chunk * Kp + (uint64_t)Np * Kp + (uint64_t)n_out * chunk) + kCrtTabBytes;
}

// f(T) with the modulus count as a compile-time constant.  No prime takes one: 1 mod 2N, it is above 2^13, and
// log2 |S| + 1.05 above 14 asks for two.
constexpr uint32_t kLeastHi32Mods = 6;  // primes from 2^40 up ask for 41 bits, five moduli hold less than 40
template <class F>
static void with_moduli(uint32_t T, F &&f) {
#define SHM_T_CASE(n) \
    case n: f(std::integral_constant<uint32_t, n>{}); break;
    switch (T) {
        SHM_T_CASE(2) SHM_T_CASE(3) SHM_T_CASE(4) SHM_T_CASE(5) SHM_T_CASE(6) SHM_T_CASE(7)
        SHM_T_CASE(8) SHM_T_CASE(9) SHM_T_CASE(10) SHM_T_CASE(11) SHM_T_CASE(12) SHM_T_CASE(13) SHM_T_CASE(14)
        SHM_T_CASE(15) SHM_T_CASE(16) SHM_T_CASE(17) SHM_T_CASE(18) SHM_T_CASE(19) SHM_T_CASE(20)
        default: throw std::invalid_argument("ct-pt matmul: modulus count out of range");
    }
#undef SHM_T_CASE
}

// Chunks of 131,072 columns run one after the other on `st`.  (Alternating them over two
// streams, so that one chunk's residue and CRT kernels could run beside the other's GEMM,
// measured no faster: the GEMM's grid fills every SM.)
void ctpt_matmul_tc(const Context &c, const uint64_t *X, const int64_t *W, uint64_t *Y, uint32_t n_in, uint32_t n_out,
                    uint32_t L, void *ws, uint64_t max_l1, cudaStream_t st) {
    if (n_in == 0 || n_out == 0) return;
    const uint64_t R = 2ull * L * c.n;
    if (R % kBN) throw std::invalid_argument("ct-pt matmul: 2 L N must be a multiple of 256");
    const uint64_t chunk = std::min<uint64_t>(R, chunk_cols());
    const uint32_t Kp = (n_in + kKB - 1) / kKB * kKB, Np = (n_out + kBM - 1) / kBM * kBM;
    Plan plan = make_plan(c, L, max_l1);
    const uint32_t T = plan.T_max;  // the weight planes and the workspaces hold T_max moduli
    SHM_CUDA(cudaMemcpyToSymbolAsync(c_mods, &plan.mods, sizeof(ModTab), 0, cudaMemcpyHostToDevice, st));
    // workspace carve-up
    uint8_t *base = static_cast<uint8_t *>(ws);
    int *err = reinterpret_cast<int *>(base);
    CrtLimb *tab = reinterpret_cast<CrtLimb *>(base + 256);
    int8_t *XP = reinterpret_cast<int8_t *>(base + kCrtTabBytes);
    int8_t *WP = XP + (size_t)T * chunk * Kp;
    uint8_t *RES = reinterpret_cast<uint8_t *>(WP + (size_t)T * Np * Kp);
    if (plan.limbs.size() > (size_t)64 * kMaxMods) throw std::invalid_argument("ct-pt matmul: too many limbs");
    SHM_CUDA(cudaMemcpyAsync(tab, plan.limbs.data(), sizeof(CrtLimb) * plan.limbs.size(), cudaMemcpyHostToDevice, st));
    SHM_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
    SHM_LAUNCHED(1);
    wres_kernel<<<dim3((Kp + 255) / 256, Np), 256, 0, st>>>(W, WP, n_in, n_out, Kp, Np, T);
    SHM_CUDA(cudaGetLastError());
    const bool resident = Kp <= kResKp;  // the X tile fits in shared memory: the persistent kernel
    CUtensorMap tmA, tmX;
    std::memset(&tmA, 0, sizeof tmA);
    std::memset(&tmX, 0, sizeof tmX);
    const bool tma_a = resident && operand_tensor_map(&tmA, WP, Kp, (uint64_t)T * Np, kBM);
    const bool limited = c.wait_limit != kSpinLimit;
    auto persistent = [limited](bool tma) {
        return limited ? (tma ? mma_persistent_kernel<true, true> : mma_persistent_kernel<false, true>)
                       : (tma ? mma_persistent_kernel<true, false> : mma_persistent_kernel<false, false>);
    };
    if (resident)
        for (const bool tma : {false, tma_a})  // a pass whose X map is refused copies its operands
            SHM_CUDA(cudaFuncSetAttribute(persistent(tma), cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemP));
    else
        SHM_CUDA(cudaFuncSetAttribute(mma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
    int sms = 0;
    SHM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device));
    const int acc_small = (uint64_t)Kp * 125 * 125 <= kAccSmall ? 1 : 0;
    bool f64_res = true;  // every limb prime below 2^51: the X residues on the FP64 pipe
    for (uint32_t l = 0; l < L; l++) f64_res = f64_res && c.primes[l] < (1ull << 51);
    for (uint64_t r0 = 0; r0 < R; r0 += chunk) {
        // a shorter last pass (2 L N not a multiple of the chunk, e.g. at N = 2^12) lays its planes out
        // with its own column count; every count here is a multiple of 256
        const uint64_t cur = std::min<uint64_t>(chunk, R - r0);
        // the pass's moduli count: the largest its limbs (rows h L + l, h = 0, 1) need
        uint32_t Tc = 0;
        for (uint64_t row = r0 >> c.log_n; row <= (r0 + cur - 1) >> c.log_n; row++)
            Tc = std::max(Tc, plan.limb_T[row % L]);
        const CrtLimb *tab_c = tab + (size_t)(Tc - plan.T_min) * L;
        SHM_LAUNCHED(1);
        const dim3 xgrid((uint32_t)(cur / (64 * kXresTiles) * (Kp / 64)));
        with_moduli(Tc, [&](auto n) {
            const auto f = f64_res ? xres_kernel<true, decltype(n)::value> : xres_kernel<false, decltype(n)::value>;
            SHM_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kXresSmem));
            f<<<xgrid, 256, kXresSmem, st>>>(X, XP, n_in, Kp, R, r0, cur);
        });
        SHM_CUDA(cudaGetLastError());
        SHM_LAUNCHED(1);
        if (resident) {
            const uint64_t tiles = (uint64_t)Tc * (cur / kBN);
            const uint32_t grid = (uint32_t)std::min<uint64_t>(tiles, (uint64_t)sms);
            // the X planes of this pass, [T * cur][Kp], as 256-row boxes (a pass's planes have its own
            // column count)
            const bool tma = tma_a && operand_tensor_map(&tmX, XP, Kp, (uint64_t)Tc * cur, kBN);
            persistent(tma)<<<grid, kThreadsP, kSmemP, st>>>(XP, WP, RES, Kp, Np, n_out, cur, Tc, err, acc_small,
                                                             c.wait_limit, tmA, tmX);
        } else {
            mma_kernel<<<dim3(Np / kBM, (uint32_t)(cur / kBN), Tc), kThreads, kSmem, st>>>(XP, WP, RES, Kp, Np, n_out,
                                                                                          cur, err, acc_small, c.wait_limit);
        }
        SHM_CUDA(cudaGetLastError());
        SHM_LAUNCHED(1);
        // 4 columns a thread; a block's columns within one limb (N and r0 are multiples of the block's)
        const uint32_t crt_threads = chunk % 1024 == 0 ? 256 : 64;
        const dim3 cgrid((uint32_t)((cur / 4 + crt_threads - 1) / crt_threads), n_out);
        with_moduli(Tc, [&](auto n) {
            constexpr uint32_t kT = decltype(n)::value;
            auto f = crt_kernel<false, kT>;
            if constexpr (kT >= kLeastHi32Mods)
                if (plan.hi32) f = crt_kernel<true, kT>;
            f<<<cgrid, crt_threads, 0, st>>>(RES, Y, tab_c, n_out, cur, r0, R, L, c.log_n, c.pc);
        });
        SHM_CUDA(cudaGetLastError());
    }
}

namespace {

// l1[o] += sum of |w_io| over 32 inputs, mx = max |w|.  Grid (n_out / 128, n_in / 32)
__global__ void weight_sums(const int64_t *__restrict__ W, uint32_t n_in, uint32_t n_out,
                            unsigned long long *__restrict__ l1, unsigned long long *__restrict__ mx) {
    const uint32_t o = blockIdx.x * 128 + threadIdx.x, i0 = blockIdx.y * 32;
    if (o >= n_out) return;
    unsigned long long s = 0, m = 0;
#pragma unroll 8
    for (uint32_t i = i0; i < min(n_in, i0 + 32); i++) {
        const int64_t w = W[(uint64_t)i * n_out + o];
        const unsigned long long a = w < 0 ? 0ull - (unsigned long long)w : (unsigned long long)w;
        s += a;
        m = a > m ? a : m;
    }
    atomicAdd(l1 + o, s);
    atomicMax(mx, m);
}

__global__ void max_sum(const unsigned long long *__restrict__ l1, uint32_t n_out, unsigned long long *__restrict__ out) {
    unsigned long long m = 0;
    for (uint32_t o = threadIdx.x; o < n_out; o += blockDim.x) m = l1[o] > m ? l1[o] : m;
    atomicMax(out, m);
}

}  // namespace

// the largest column sum of |W| (below n_in 2^40) and the largest |W|; uses the plane area of ws
void ctpt_weight_norms(const int64_t *W, uint32_t n_in, uint32_t n_out, void *ws, uint64_t &max_l1, uint64_t &max_w,
                       cudaStream_t st) {
    auto *t = reinterpret_cast<unsigned long long *>(static_cast<uint8_t *>(ws) + kCrtTabBytes);  // max w, max l1, l1[]
    SHM_CUDA(cudaMemsetAsync(t, 0, ((size_t)n_out + 2) * 8, st));
    SHM_LAUNCHED(2);
    weight_sums<<<dim3((n_out + 127) / 128, (n_in + 31) / 32), 128, 0, st>>>(W, n_in, n_out, t + 2, t);
    max_sum<<<1, 256, 0, st>>>(t + 2, n_out, t + 1);
    SHM_CUDA(cudaGetLastError());
    uint64_t h[2];
    SHM_CUDA(cudaMemcpyAsync(h, t, sizeof h, cudaMemcpyDeviceToHost, st));
    SHM_CUDA(cudaStreamSynchronize(st));
    max_w = h[0];
    max_l1 = h[1];
}

int ctpt_tc_error(void *ws, cudaStream_t st) {
    int h = 0;
    SHM_CUDA(cudaMemcpyAsync(&h, ws, sizeof(int), cudaMemcpyDeviceToHost, st));
    SHM_CUDA(cudaStreamSynchronize(st));
    return h;
}

}  // namespace shm

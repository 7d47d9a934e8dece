// Dispatch of the NTT launches over the ring and the butterfly families; the kernels are instantiated
// in ntt_n12_*.cu and ntt_n16_*.cu.
#include "ntt_kernels.cuh"

namespace shm {

#define SHM_NTT_EXTERN(R, FAM)                                                                                    \
    extern template void launch_fwd<R, FAM>(const Context &, int, uint64_t *, const NttRows &, cudaStream_t,     \
                                            const NttIO &);                                                       \
    extern template void launch_inv<R, FAM>(const Context &, const InvArgs &, const NttRows &, cudaStream_t);
SHM_NTT_EXTERN(3, kFamSmall)
SHM_NTT_EXTERN(3, kFamLarge)
SHM_NTT_EXTERN(3, kFamAll)
SHM_NTT_EXTERN(4, kFamSmall)
SHM_NTT_EXTERN(4, kFamLarge)
SHM_NTT_EXTERN(4, kFamAll)

namespace {

// f(ring, families) with both as compile-time constants
template <class F>
void dispatch(const Context &c, F &&f) {
    using std::integral_constant;
    auto fam = [&](auto r) {
        switch (c.ntt_families) {
            case kFamSmall: f(r, integral_constant<int, kFamSmall>{}); break;
            case kFamLarge: f(r, integral_constant<int, kFamLarge>{}); break;
            default: f(r, integral_constant<int, kFamAll>{}); break;
        }
    };
    if (c.log_n == 16) fam(integral_constant<int, 4>{});
    else if (c.log_n == 12) fam(integral_constant<int, 3>{});
    else throw std::invalid_argument("NTT supports N = 2^12 and 2^16");
    SHM_CUDA(cudaGetLastError());
}

void forward(const Context &c, int kind, uint64_t *data, const NttRows &rw, cudaStream_t st, const NttIO &io = {}) {
    if (rw.polys == 0 || rw.count == 0) return;
    dispatch(c, [&](auto r, auto fam) { launch_fwd<decltype(r)::value, decltype(fam)::value>(c, kind, data, rw, st, io); });
}

}  // namespace

NttRows rows_of(const Context &c, uint32_t polys, uint32_t slots, uint32_t lq) {
    NttRows r;
    r.polys = polys;
    r.slots = r.count = r.lp = slots;
    r.lq = lq;
    r.nq = c.nq;
    return r;
}

void ntt_forward(const Context &c, uint64_t *data, const NttRows &rw, cudaStream_t st) {
    forward(c, kIoPlain, data, rw, st);
}

void ntt_forward_rescale(const Context &c, const RescaleIO &rs, uint64_t *t, uint32_t n_polys, uint32_t L,
                         cudaStream_t st) {
    NttIO io;
    io.rs = rs;
    forward(c, kIoRescale, t, rows_of(c, n_polys, L - 1, L - 1), st, io);
}

void ntt_forward_moddown(const Context &c, const ModDownIO &md, uint64_t *delta, uint32_t n_polys, uint32_t L,
                         cudaStream_t st) {
    if (n_polys == 0) return;
    if (md.np > 16 || md.H == 0) throw std::invalid_argument("ModDown: shape out of range");
    NttIO io;
    io.md = md;
    if (md.bytes) {
        ConvIO cv;
        cv.src = md.acc + (size_t)L * c.n;
        cv.src_ct = (size_t)(L + md.np) * c.n;
        cv.bytes = md.bytes;
        cv.out = delta;
        cv.vrow = md.vrow;
        cv.sets = n_polys;
        cv.na = cv.total = md.np;
        cv.rows = cv.lq = L;
        conv_rows(c, cv, st);
        io.converted = 1;
    }
    forward(c, kIoModDown, delta, rows_of(c, n_polys, L, L), st, io);
}

void ntt_forward_modup(const Context &c, const ModUpIO &mu, uint64_t *up, uint32_t n_cts, uint32_t beta,
                       cudaStream_t st) {
    if (n_cts == 0) return;
    if (mu.np > 16 || mu.np == 0 || mu.LP != mu.L + mu.np) throw std::invalid_argument("ModUp: shape out of range");
    NttIO io;
    io.mu = mu;
    NttRows rw = rows_of(c, n_cts, beta * mu.LP, mu.L);
    rw.lp = mu.LP;
    rw.skip = mu.np;
    if (mu.bytes) {
        ConvIO cv;
        cv.src = mu.x;
        cv.src_ct = (size_t)mu.L * c.n;
        cv.bytes = mu.bytes;
        cv.out = up;
        cv.skip_own = true;
        cv.sets = n_cts * beta;
        cv.per = beta;
        cv.na = mu.np;
        cv.total = mu.L;
        cv.rows = mu.LP;
        cv.lq = mu.L;
        cv.nq = c.nq;
        conv_rows(c, cv, st);
        io.converted = 1;
    }
    forward(c, kIoModUp, up, rw, st, io);
}

void ntt_inverse(const Context &c, uint64_t *data, const NttRows &rw, const uint64_t *scale, cudaStream_t st,
                 const uint64_t *src, size_t src_stride) {
    if (rw.polys == 0 || rw.count == 0) return;
    const InvArgs v{data, src ? src : data, src ? src_stride : (size_t)rw.slots * c.n, scale};
    dispatch(c, [&](auto r, auto fam) { launch_inv<decltype(r)::value, decltype(fam)::value>(c, v, rw, st); });
}

}  // namespace shm

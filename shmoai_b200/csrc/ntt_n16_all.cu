#include "ntt_kernels.cuh"

namespace shm {

template void launch_fwd<4, kFamAll>(const Context &, int, uint64_t *, const NttRows &, cudaStream_t, const NttIO &);
template void launch_inv<4, kFamAll>(const Context &, const InvArgs &, const NttRows &, cudaStream_t);

}  // namespace shm

#include "ntt_kernels.cuh"

namespace shm {

template void launch_fwd<3, kFamLarge>(const Context &, int, uint64_t *, const NttRows &, cudaStream_t, const NttIO &);
template void launch_inv<3, kFamLarge>(const Context &, const InvArgs &, const NttRows &, cudaStream_t);

}  // namespace shm

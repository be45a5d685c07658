// align_k8.cu -- the batched round's kernels for tables of 8 entries.
#include "align_round.cuh"

namespace ngia {

template int launch_align_k<8>(int kernel, const RoundArgs &a, uint32_t m, cudaStream_t s);

}  // namespace ngia

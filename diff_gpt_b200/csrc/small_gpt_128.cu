// dgpt_small_gpt, models 128 wide (see small_gpt.cu)
#include "small_gpt.cuh"

namespace dgpt {

int small_gpt_128(const SmallGpt& p, int M, int grid, cudaStream_t st) { return small_gpt_pick<128>(p, M, grid, st); }

}  // namespace dgpt

// Stage 1 for 2 local kv heads
#include "ommx_stage1.cuh"

int ommx::launch_stage1_h2(const S1Params &p, size_t smem, cudaStream_t st) { return launch_s1_heads<2>(p, smem, st); }

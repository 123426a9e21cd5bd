// Stage 1 for 4 local kv heads
#include "ommx_stage1.cuh"

int ommx::launch_stage1_h4(const S1Params &p, size_t smem, cudaStream_t st) { return launch_s1_heads<4>(p, smem, st); }

// Stage 1 for 1 local kv head
#include "ommx_stage1.cuh"

int ommx::launch_stage1_h1(const S1Params &p, size_t smem, cudaStream_t st) { return launch_s1_heads<1>(p, smem, st); }

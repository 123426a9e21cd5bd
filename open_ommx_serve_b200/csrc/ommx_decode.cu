// Paged decode attention over OMMX-quantized KV planes for sm_100a: split-KV stage 1, stage 2
// (log-sum-exp combine with the bf16 sink/recent rows fused in) and the partial-state merge.
//
// Stage 1 (ommx_stage1.cuh) replaces _canonical_splitkv_stage1 (ommx_gpu_serve/attention/paged_decode.py:1255-2284
// of the reference).  The groups of all sequences form one running list of which every CTA takes a
// contiguous share, for ALL local kv heads, so every page row it touches is a full contiguous line:
//
//   producer warp   streams whole pages / group-slot planes into a shared-memory ring: the two
//                   code planes through swizzled tensor maps, the small planes with 1-D bulk
//                   copies, completion through mbarrier transaction counts; page ids and group
//                   slots are read one ring stage ahead.
//   15 decode warps build, two per (group, kv head) unit, the unit's sidecar tile: outlier
//                   deltas (bit walk, FP4 nibble, base code) as bf16
//                   [token][channel], and the power-of-two K and V scale factors laid out in
//                   MMA-fragment order.
//   8 MMA warps     own one unit per stage and a private online-softmax state.  All MMAs are
//                   m16n8k16 with the 2-bit codes as the A operand - a code field masked in
//                   place is a subnormal, exact and offset-free, in bf16 for the logits and in
//                   fp16 for the output - and
//                   the query heads as the 8 columns: logits = codes.(q*2^e) + delta.q + q.zp,
//                   softmax over token rows, P transposed with movmatrix, output =
//                   codes^T.(P*2^e_v) + vz^T.P.
//
// Numerics follow the reference kernel's rounding points: q*sm_scale rounded to bf16, exact
// code*2^e products, the outlier delta rounded to bf16, q.zp as an fp32 dot product of the raw
// query with the zero-points (paged_decode.py:1754-1770), fp32 accumulation, V as exact code*2^e
// products with the zero-point bias summed apart.  One point differs inside the gate: P is rounded
// to fp16 (11 bits) instead of bf16.
#include "ommx_stage1.cuh"

#include <new>
#include <unordered_map>

namespace ommx {

// =================================================================================================
// Stage 2: bf16 sink/recent rows + log-sum-exp combine (reference: paged_decode.py:2366-2500)
// =================================================================================================
struct S2Params {
    const __nv_bfloat16 *q;
    int64_t q_sb, q_sh;
    int32_t Hq, gqa, D;
    const __nv_bfloat16 *k_tail, *v_tail;
    int64_t t_sb, t_st, t_sh;
    const int32_t *b_tail_len, *b_seq_len;
    int32_t max_tail, v_vec_ok;          // v_vec_ok: four adjacent V elements may be fetched as one 8-byte word
    const float *al;
    int64_t al_sb, al_sh, al_ss;
    int32_t S, B;
    Stage1Grid grid;                     // stage 1's launch; ncta = 0: equal splits per sequence
    ShareDivisors by;                    // of it
    void *o;
    int32_t o_bf16;
    int64_t o_sb, o_sh;
    float *lse;
    int64_t lse_sb;
    float sm_scale, logit_cap;
    // head-output exchange (g_world <= 1: none)
    int32_t g_world, g_rank;
    uint64_t *const *g_recv;
    float *g_out;
    uint32_t *g_state;
    int32_t *status;
};

__device__ __forceinline__ float warp_max(float x) {                     // over the lanes; a NaN is ignored where there is anything else
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
    return r;
}
typedef void (*Stage2Kernel)(S2Params);
constexpr int S2_MAX_TAIL = 256;
constexpr int S2_MAX_SPLITS = 1024;

// One CTA per (query head, sequence).  Warps stripe over the bf16 residual rows, then over the splits for the combine; every loop keeps
// many independent loads in flight.  Few rows are a chain of round trips (lengths, residual rows, splits: 64 KB to an SM at 127 splits),
// many are bound by instruction issue too, so the divisions of the share-out are multiplications by what the host prepared and lie
// where the residual rows are on their way, and a warp's maximum is one instruction.  Both stages, us a layer in a graph, with three
// divisions ahead of the loads and maxima by exchanges -> now, 8 kv heads: 32 rows 4K 11.0 -> 10.6, 16K 18.5 -> 18.0; at 1835 tokens 64
// rows 11.6 -> 11.0, 128 15.1 -> 14.4, 256 19.5 -> 18.8, 704 23.9 -> 23.2, 1280 33.3 -> 32.3, 2048 50.6 -> 49.2; 512 rows 4K 28.1 -> 27.2.
// Requesting the splits before the residual rows are worked in helps where a block starts late and costs as much where it waits
// early (1K 8.8 -> 10.3).  Logits by MMA took fewer instructions, but the sum of sixteen products is cut off where a
// multiply-add rounds (logits 5 % further from 64 bits), and eight rows to a batch made turns of 32 rows (704 rows 24.8, 1280 35.7, 2048 52.3).
// Four sizes (NW warps, PER_SM blocks to an SM), by what the rows of the grid need to run side by side (chosen in
// launch_stage2): the more warps a row can have, the more of its loads are in flight at once, but a second round of blocks
// costs more than that gains (4K, 32 rows: 16 warps 12.5 us, 8 warps 13.9, 4 warps 15.6).
// CLUSTER: stage 1 was launched in clusters.  Choosing between its two plans in every launch cost 0.1 us (32 layers at 4K 389 -> 392 us).
template <int NW, int PER_SM, bool CLUSTER>
__global__ void __launch_bounds__(NW * 32, PER_SM) decode_stage2_kernel(const S2Params p) {
    __shared__ __align__(16) float s_q[HD];
    __shared__ float s_w[NW], s_red[NW];
    __shared__ __align__(16) float s_acc[NW][HD];
    // the next kernel in the stream (the following layer's stage 1) may be placed as SMs free up; it waits for
    // this grid to finish before it touches memory
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int hq = blockIdx.x, b = blockIdx.y;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kvh = hq / p.gqa;
    int tail = p.b_tail_len ? p.b_tail_len[b] : 0;                       // requested before the lengths are waited for
    // Lengths: this sequence's, and what the share-out of stage 1 depends on (all, longest, those before this one), in one
    // round of loads.
    const int groups = groups_of(p.b_seq_len[b]);
    int total = groups, longest = groups, before = 0;
    if (p.B > 1) {
        total = 0;
        for (int i = lane; i < p.B; i += 32) {
            const int n = groups_of(p.b_seq_len[i]);
            total += n;
            longest = max(longest, n);
            if (i < b) before += n;
        }
        total = __reduce_add_sync(0xFFFFFFFFu, total);
        before = __reduce_add_sync(0xFFFFFFFFu, before);
        longest = __reduce_max_sync(0xFFFFFFFFu, longest);
    }
    tail = max(0, min(tail, min(p.max_tail, S2_MAX_TAIL)));
    const int D = p.D;                                                   // == HD

    // workspace slots stage 1 wrote for this sequence: worked out while the residual rows are on their way
    int nsplit = 0;
    auto count_splits = [&]() __attribute__((always_inline)) {
        if (p.S > 0 && groups > 0) {
            int per = 0;
            if constexpr (CLUSTER) per = share_plan_of(total, longest, p.B, p.S, p.grid, p.by).per;
            else if (p.grid.ncta > 0) per = share_plan_of(total, longest, p.B, p.S, p.by.ctas, p.grid.waves, p.by).per;
            if (per == 0) {
                const int equal = p.by.slots.of(groups + p.S - 1);
                nsplit = (groups + equal - 1) / equal;
            } else {
                nsplit = (before + groups - 1) / per + 1;
                if (before > 0) nsplit -= before / per;
            }
        }
    };
    // ---- bf16 residual rows of this q head: they do not depend on stage 1, so everything about them happens before its end is
    //      waited for ----
    // A warp takes rows warp, warp + NW, ..., four of them to a batch for the logits: eight lanes to a row, sixteen channels to a lane, three
    // exchanges for four rows; and KB such batches in a turn of the loop, and the next turn takes over the softmax state.  The rows a
    // window usually has (8 + 32 + up to 31) are one turn, or two (of 48) where seven blocks share an SM's registers.
    constexpr int KB = NW == 16 ? 2 : (PER_SM == 4 ? 5 : 3), ROWS = 4 * KB;
    constexpr int V_FIRST = PER_SM == 1 ? ROWS : (PER_SM <= 4 ? ROWS / 2 : ROWS / 4);   // the registers of the K rows hold the others
    float m_t = -INFINITY, den_t = 0.f, v0 = 0.f, v1 = 0.f, v2 = 0.f, v3 = 0.f;    // v: channels 4 lane .. 4 lane + 3
    if (tail > 0) {
        const __nv_bfloat16 *kt = p.k_tail + (int64_t)b * p.t_sb + (int64_t)kvh * p.t_sh + 4 * (lane & 7);
        const __nv_bfloat16 *vt = p.v_tail + (int64_t)b * p.t_sb + (int64_t)kvh * p.t_sh + 4 * lane + (int64_t)warp * p.t_st;
        const int64_t v_step = (int64_t)NW * p.t_st;
        float q_own = 0.f;
        if (tid < D) q_own = __bfloat162float(p.q[(int64_t)b * p.q_sb + (int64_t)hq * p.q_sh + tid]);
#pragma unroll 1
        for (int r0 = warp; r0 - warp < tail; r0 += NW * ROWS) {
            uint2 kx[KB][4], vx[ROWS];                                   // K: channels 4 (lane % 8) + 32 i of row lane / 8 of the batch
#pragma unroll
            for (int k = 0; k < KB; ++k) {
                const int r = r0 + NW * (4 * k + (lane >> 3));
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    kx[k][i] = make_uint2(0u, 0u);
                    if (r < tail) kx[k][i] = *reinterpret_cast<const uint2 *>(kt + (int64_t)r * p.t_st + 32 * i);
                }
            }
            auto load_v = [&](int k) __attribute__((always_inline)) {
                vx[k] = make_uint2(0u, 0u);
                if (r0 + NW * k >= tail) return;
                const __nv_bfloat16 *row = vt + k * v_step;
                if (p.v_vec_ok) vx[k] = *reinterpret_cast<const uint2 *>(row);
                else {
                    const uint16_t *e = reinterpret_cast<const uint16_t *>(row);
                    vx[k] = make_uint2(e[0] | ((uint32_t)e[1] << 16), e[2] | ((uint32_t)e[3] << 16));
                }
            };
#pragma unroll
            for (int k = 0; k < V_FIRST; ++k) load_v(k);
            if (r0 == warp) {
                count_splits();
                if (tid < D) s_q[tid] = q_own;
                __syncthreads();
            }
            float x[KB], mx = -INFINITY;
#pragma unroll
            for (int k = 0; k < KB; ++k) x[k] = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 q = *reinterpret_cast<const float4 *>(s_q + 4 * (lane & 7) + 32 * i);
#pragma unroll
                for (int k = 0; k < KB; ++k) {
                    float t = q.x * bf16_bits_to_f32(kx[k][i].x & 0xFFFFu);            // (the product of two bf16 values is exact)
                    t = __fmaf_rn(q.y, bf16_bits_to_f32(kx[k][i].x >> 16), t);
                    t = __fmaf_rn(q.z, bf16_bits_to_f32(kx[k][i].y & 0xFFFFu), t);
                    x[k] = __fadd_rn(x[k], __fmaf_rn(q.w, bf16_bits_to_f32(kx[k][i].y >> 16), t));
                }
            }
#pragma unroll
            for (int k = V_FIRST; k < ROWS; ++k) load_v(k);
#pragma unroll
            for (int k = 0; k < KB; ++k) {
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) x[k] += __shfl_xor_sync(0xFFFFFFFFu, x[k], o);
                x[k] *= p.sm_scale;
                if (p.logit_cap > 0.f) x[k] = p.logit_cap * tanhf(x[k] / p.logit_cap);
                if (r0 + NW * (4 * k + (lane >> 3)) >= tail) x[k] = -INFINITY;
                mx = fmaxf(mx, x[k]);
            }
            const float m_new = fmaxf(m_t, warp_max(mx)), m_use = (m_new == -INFINITY) ? 0.f : m_new, corr = __expf(m_t - m_use);
            m_t = m_new;
            den_t *= corr; v0 *= corr; v1 *= corr; v2 *= corr; v3 *= corr;
#pragma unroll
            for (int k = 0; k < KB; ++k) x[k] = __expf(x[k] - m_use);    // 0 for the rows past the end
#pragma unroll
            for (int k = 0; k < ROWS; ++k) {
                const float w = __shfl_sync(0xFFFFFFFFu, x[k >> 2], 8 * (k & 3));
                den_t += w;
                v0 += w * bf16_bits_to_f32(vx[k].x & 0xFFFFu); v1 += w * bf16_bits_to_f32(vx[k].x >> 16);
                v2 += w * bf16_bits_to_f32(vx[k].y & 0xFFFFu); v3 += w * bf16_bits_to_f32(vx[k].y >> 16);
            }
            vt += ROWS * v_step;
        }
    } else {
        count_splits();
    }
    // the channels lane + 32 i, as the rows of the splits are read
    *reinterpret_cast<float4 *>(&s_acc[warp][4 * lane]) = make_float4(v0, v1, v2, v3);
    __syncwarp();
    float a0 = s_acc[warp][lane], a1 = s_acc[warp][lane + 32], a2 = s_acc[warp][lane + 64], a3 = s_acc[warp][lane + 96];
    // ---- everything below reads what stage 1 wrote: wait for that grid (no-op without a
    //      programmatic launch) ----
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // Every warp folds its own splits (warp, warp + NW, ...) into its softmax state of the residual rows - maximum, sum of
    // weights, weighted rows - with no exchange: the lse of a split is read by all lanes at once (one address).  The NW states are
    // merged once at the end.  The split rows are requested together with the lse values, not after the weights are
    // known: the kernel is a chain of global round trips and this takes one link out of it.
    constexpr int PRE_S = NW == 16 ? 10 : 5;                              // splits per warp held in registers
    const float *base = p.al + (int64_t)b * p.al_sb + (int64_t)hq * p.al_sh;
    float spre[PRE_S][4], lpre[PRE_S];
#pragma unroll
    for (int k = 0; k < PRE_S; ++k) {
        const int s = warp + k * NW;
        spre[k][0] = spre[k][1] = spre[k][2] = spre[k][3] = 0.f;
        lpre[k] = -INFINITY;
        if (s < nsplit) {
            const float *row = base + (int64_t)s * p.al_ss;
            spre[k][0] = row[lane]; spre[k][1] = row[lane + 32]; spre[k][2] = row[lane + 64]; spre[k][3] = row[lane + 96];
            lpre[k] = row[D];
        }
    }
    float m_w = m_t;
#pragma unroll
    for (int k = 0; k < PRE_S; ++k) m_w = fmaxf(m_w, lpre[k]);
    for (int s = warp + PRE_S * NW; s < nsplit; s += NW) m_w = fmaxf(m_w, base[(int64_t)s * p.al_ss + D]);
    const float m_safe = (m_w == -INFINITY) ? 0.f : m_w;
    // weighted sum: lane owns channels lane + 32*i
    const float f_t = __expf(m_t - m_safe);                               // 0 without residual rows
    float den_w = den_t * f_t;
    a0 *= f_t; a1 *= f_t; a2 *= f_t; a3 *= f_t;
#pragma unroll
    for (int k = 0; k < PRE_S; ++k) {
        const float w = __expf(lpre[k] - m_safe);                        // exp(-inf) = 0 for the slots past nsplit
        den_w += w;
        a0 += w * spre[k][0]; a1 += w * spre[k][1]; a2 += w * spre[k][2]; a3 += w * spre[k][3];
    }
#pragma unroll 4
    for (int s = warp + PRE_S * NW; s < nsplit; s += NW) {
        const float *row = base + (int64_t)s * p.al_ss;
        const float w = __expf(row[D] - m_safe);
        den_w += w;
        a0 += w * row[lane]; a1 += w * row[lane + 32]; a2 += w * row[lane + 64]; a3 += w * row[lane + 96];
    }
    s_acc[warp][lane] = a0; s_acc[warp][lane + 32] = a1;
    s_acc[warp][lane + 64] = a2; s_acc[warp][lane + 96] = a3;
    if (lane == 0) { s_red[warp] = m_w; s_w[warp] = den_w; }
    __syncthreads();
    // ---- merge of the NW states ----
    float out = 0.f;
    if (tid < D) {
        float g_max = s_red[0];
#pragma unroll
        for (int w = 1; w < NW; ++w) g_max = fmaxf(g_max, s_red[w]);
        const float g_safe = (g_max == -INFINITY) ? 0.f : g_max;
        float acc = 0.f, den = 0.f;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            const float e = __expf(s_red[w] - g_safe);                   // 0 for a warp that saw nothing
            acc = fmaf(s_acc[w][tid], e, acc);
            den = fmaf(s_w[w], e, den);
        }
        out = acc / (den > 0.f ? den : 1.f);
        if (p.o_bf16) reinterpret_cast<__nv_bfloat16 *>(p.o)[(int64_t)b * p.o_sb + (int64_t)hq * p.o_sh + tid] = __float2bfloat16_rn(out);
        else reinterpret_cast<float *>(p.o)[(int64_t)b * p.o_sb + (int64_t)hq * p.o_sh + tid] = out;
        if (tid == 0) p.lse[(int64_t)b * p.lse_sb + hq] = g_max + logf(den);
    }
    if (p.g_world > 1) {
        // Sharded heads: the row travels to every peer as 8-byte words (value, call count); a word arrives whole,
        // so the count tells the receiver that the value beside it is this call's.  Then this block collects the
        // same row of every peer from its own receive buffer.
        __shared__ uint32_t s_epoch;
        if (tid == 0) s_epoch = *reinterpret_cast<volatile uint32_t *>(&p.g_state[0]) + 1u;
        __syncthreads();
        const uint32_t epoch = s_epoch;
        const int64_t slot = (int64_t)gridDim.y * p.Hq * D;            // elements of one rank's slot
        const int64_t row = ((int64_t)b * p.Hq + hq) * D;
        if (tid < D) {
            const uint64_t word = ((uint64_t)epoch << 32) | (uint64_t)__float_as_uint(out);
            for (int r = 0; r < p.g_world; ++r)
                if (r != p.g_rank)
                    asm volatile("st.volatile.global.u64 [%0], %1;" ::"l"(p.g_recv[r] + (int64_t)p.g_rank * slot + row + tid), "l"(word) : "memory");
            p.g_out[(int64_t)p.g_rank * slot + row + tid] = out;
        }
        const uint64_t *mine = p.g_recv[p.g_rank];
        const long long t_end = clock64() + WAIT_LIMIT_CYCLES;
        const int n_words = (p.g_world - 1) * D;
        // two words per thread and round, both requested before either is looked at
        for (int idx = tid; idx < n_words; idx += 2 * (NW * 32)) {
            const uint64_t *src[2];
            float *dst[2];
            bool pending[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int i = idx + u * (NW * 32);
                pending[u] = i < n_words;
                int r = pending[u] ? i / D : 0;
                const int e = pending[u] ? i - r * D : 0;
                r += (r >= p.g_rank) ? 1 : 0;                          // skip the own slot
                src[u] = mine + (int64_t)r * slot + row + e;
                dst[u] = p.g_out + (int64_t)r * slot + row + e;
            }
            for (uint32_t i = 1; pending[0] || pending[1]; ++i) {
                uint64_t word[2] = {0, 0};
#pragma unroll
                for (int u = 0; u < 2; ++u)
                    if (pending[u]) asm volatile("ld.volatile.global.u64 %0, [%1];" : "=l"(word[u]) : "l"(src[u]) : "memory");
#pragma unroll
                for (int u = 0; u < 2; ++u)
                    if (pending[u] && (uint32_t)(word[u] >> 32) == epoch) {
                        *dst[u] = __uint_as_float((uint32_t)word[u]);
                        pending[u] = false;
                    }
                if ((i & 63u) == 0 && clock64() > t_end) { or_status(p.status, OMMX_ST_TIMEOUT); break; }
            }
        }
        // the call count moves on once every block has read it: each block reads it before it draws its ticket
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            const uint32_t t = atomicAdd(&p.g_state[1], 1u);
            if (t == gridDim.x * gridDim.y - 1u) {
                p.g_state[1] = 0u;
                p.g_state[0] = epoch;
            }
        }
    }
}

// =================================================================================================
// merge of partial softmax states (reference: paged_decode.py:2650-2690)
// =================================================================================================
__global__ void __launch_bounds__(128) merge_states_kernel(const float *o_parts, const float *lse_parts,
                                                           const int32_t *valid, int P, int R, int D,
                                                           float *o, float *lse) {
    const int r = blockIdx.x;
    int np = P;
    if (valid) { int v = valid[r]; if (v >= 0) np = min(v, P); }
    float m = -INFINITY;
    for (int q = 0; q < np; ++q) m = fmaxf(m, lse_parts[(int64_t)q * R + r]);
    const float ms = (m == -INFINITY) ? 0.f : m;
    float den = 0.f;
    for (int q = 0; q < np; ++q) den += __expf(lse_parts[(int64_t)q * R + r] - ms);
    for (int d = threadIdx.x; d < D; d += blockDim.x) {
        float acc = 0.f;
        for (int q = 0; q < np; ++q)
            acc += __expf(lse_parts[(int64_t)q * R + r] - ms) * o_parts[((int64_t)q * R + r) * D + d];
        o[(int64_t)r * D + d] = acc / (den > 0.f ? den : 1.f);
    }
    if (threadIdx.x == 0) lse[r] = ms + logf(den);
}

// =================================================================================================
// host side
// =================================================================================================
static int validate_decode(const ommx_decode_args *a) {
    if (!a) return fail(OMMX_E_ARG, "decode: null args");
    const ommx_kv_planes &pl = a->planes;
    if (!a->q || !a->o || !a->lse || !a->attn_logits || !a->b_seq_len)
        return fail(OMMX_E_ARG, "decode: q/o/lse/attn_logits/b_seq_len must not be null");
    if (a->q_dtype != OMMX_DT_BF16) return fail(OMMX_E_UNSUPPORTED, "decode: q must be bf16");
    if (a->o_dtype != OMMX_DT_F32 && a->o_dtype != OMMX_DT_BF16) return fail(OMMX_E_UNSUPPORTED, "decode: o must be f32 or bf16");
    if (pl.head_dim != HD) return fail(OMMX_E_UNSUPPORTED, "decode: head_dim=%d (this build serves %d)", pl.head_dim, HD);
    if (pl.n_kv_heads != 1 && pl.n_kv_heads != 2 && pl.n_kv_heads != 4 && pl.n_kv_heads != 8)
        return fail(OMMX_E_UNSUPPORTED, "decode: n_kv_heads=%d per device must be 1, 2, 4 or 8", pl.n_kv_heads);
    if (a->batch <= 0 || a->n_q_heads <= 0 || a->n_q_heads % pl.n_kv_heads != 0)
        return fail(OMMX_E_ARG, "decode: batch=%d n_q_heads=%d n_kv_heads=%d", a->batch, a->n_q_heads, pl.n_kv_heads);
    if (a->n_q_heads / pl.n_kv_heads > 8)
        return fail(OMMX_E_UNSUPPORTED, "decode: GQA group of %d query heads per kv head (max 8)", a->n_q_heads / pl.n_kv_heads);
    if (pl.page_size != 8 && pl.page_size != 16 && pl.page_size != 32)
        return fail(OMMX_E_UNSUPPORTED, "decode: page_size=%d must be 8, 16 or 32", pl.page_size);
    if (pl.scale_kind != OMMX_SCALE_INT8_EXP)
        return fail(OMMX_E_UNSUPPORTED, "decode: only int8 power-of-two scale planes are served (pack with use_pow2)");
    if (pl.outliers_per_vector < 0 || pl.outliers_per_vector > 16)
        return fail(OMMX_E_UNSUPPORTED, "decode: outliers_per_vector=%d outside [0,16]", pl.outliers_per_vector);
    if (pl.outlier_index != OMMX_OIDX_BITMASK && pl.outlier_index != OMMX_OIDX_RELIDX7)
        return fail(OMMX_E_ARG, "decode: outlier_index=%d", pl.outlier_index);
    if (pl.outlier_index == OMMX_OIDX_RELIDX7 && (128 * ((7 * pl.outliers_per_vector + 7) / 8)) % 16 != 0)
        return fail(OMMX_E_UNSUPPORTED, "decode: relidx7 frames of %d outliers do not stage in 16-byte pieces", pl.outliers_per_vector);
    if (a->packed_start_offset != 0) return fail(OMMX_E_UNSUPPORTED, "decode: packed_start_offset must be 0");
    if (a->seg_group_base < 0) return fail(OMMX_E_ARG, "decode: seg_group_base=%d", a->seg_group_base);
    if (a->num_kv_splits < 1) return fail(OMMX_E_ARG, "decode: num_kv_splits=%d", a->num_kv_splits);
    if (a->num_kv_splits > S2_MAX_SPLITS) return fail(OMMX_E_UNSUPPORTED, "decode: num_kv_splits=%d (max %d)", a->num_kv_splits, S2_MAX_SPLITS);
    if (a->max_tail_len > S2_MAX_TAIL) return fail(OMMX_E_UNSUPPORTED, "decode: max_tail_len=%d (max %d)", a->max_tail_len, S2_MAX_TAIL);
    if (a->max_tail_len > 0 && (!a->k_tail || !a->v_tail || !a->b_tail_len))
        return fail(OMMX_E_ARG, "decode: max_tail_len>0 needs k_tail, v_tail and b_tail_len");
    // stage 2 reads K rows in 8-byte words; a stride that no index goes along may be anything
    if (a->max_tail_len > 0 && (((uintptr_t)a->k_tail & 7) != 0 || (a->batch > 1 && a->tail_stride_b % 4 != 0) ||
                                (a->max_tail_len > 1 && a->tail_stride_t % 4 != 0) || (pl.n_kv_heads > 1 && a->tail_stride_h % 4 != 0)))
        return fail(OMMX_E_ARG, "decode: k_tail rows must start on 8-byte boundaries (base %% 8 = %d bytes, strides %lld, %lld, %lld elements)",
                    (int)((uintptr_t)a->k_tail & 7), (long long)a->tail_stride_b, (long long)a->tail_stride_t, (long long)a->tail_stride_h);
    if (a->max_seq_len > 0) {
        if (!a->req_to_token || !a->req_to_group) return fail(OMMX_E_ARG, "decode: page / group tables are null");
        if (!pl.k_base || !pl.k_scale || !pl.k_zp || !pl.v_main || !pl.v_scale || !pl.v_zp)
            return fail(OMMX_E_ARG, "decode: a KV plane is null");
        if (pl.outliers_per_vector > 0 && (!pl.k_obmp || !pl.k_oval))
            return fail(OMMX_E_ARG, "decode: k>0 needs k_obmp and k_oval");
        if (pl.outliers_per_vector > 0 && pl.kv_outlier_map && (!pl.k_mapscale || !pl.k_mapcenter))
            return fail(OMMX_E_ARG, "decode: kv_outlier_map needs k_mapscale and k_mapcenter");
        const void *pp[] = {pl.k_base, pl.k_scale, pl.k_zp, pl.k_obmp, pl.k_oval, pl.k_mapscale, pl.k_mapcenter,
                            pl.v_main, pl.v_scale, pl.v_zp};
        for (const void *x : pp)
            if (((uintptr_t)x & 15) != 0) return fail(OMMX_E_ARG, "decode: every KV plane must be 16-byte aligned");
        const int min_s = ommx_b200_min_num_kv_splits(a->max_seq_len, pl.page_size);
        if (a->num_kv_splits < min_s)
            return fail(OMMX_E_ARG, "decode: num_kv_splits=%d too small for max_seq_len=%d (need >= %d)",
                        a->num_kv_splits, a->max_seq_len, min_s);
    }
    if (a->al_stride_s < HD + 1) return fail(OMMX_E_ARG, "decode: attn_logits last dim must be head_dim+1");
    return 0;
}

// ---- tensor maps of the code planes (driver entry point looked up at run time, no link dependency) ----
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_tiled_fn() {
    static std::atomic<int> state{0};                 // 0 unknown, 1 found, 2 absent
    static EncodeTiledFn fn = nullptr;
    int st = state.load(std::memory_order_acquire);
    if (st == 0) {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        const bool ok = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess &&
                        q == cudaDriverEntryPointSuccess && f != nullptr;
        if (ok) fn = reinterpret_cast<EncodeTiledFn>(f);
        (void)cudaGetLastError();
        state.store(ok ? 1 : 2, std::memory_order_release);
        st = ok ? 1 : 2;
    }
    return st == 1 ? fn : nullptr;
}

static std::atomic<long long> g_map_encodings{0};

// box_rows > 0: the plane viewed as [bytes/128][128] uint8, box = one page, 128-byte swizzle.  box_rows = 0: the plane viewed as
// [bytes/row_bytes][row_bytes], box = one row as it lies (for loads of four rows).  Returns false when the map cannot be built.
static bool encode_map(CUtensorMap *m, const void *base, int64_t total_bytes, int row_bytes, int box_rows) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (fn == nullptr || total_bytes < row_bytes || row_bytes % 16 != 0 || row_bytes > GATHER_ROW_MAX || box_rows > 256) return false;
    // a box is at most 256 elements wide
    const int element = row_bytes <= 256 ? 1 : (row_bytes <= 1024 ? 4 : 8);
    const CUtensorMapDataType type = element == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : (element == 4 ? CU_TENSOR_MAP_DATA_TYPE_INT32 : CU_TENSOR_MAP_DATA_TYPE_INT64);
    cuuint64_t gdim[2] = {(cuuint64_t)(row_bytes / element), (cuuint64_t)(total_bytes / row_bytes)};
    cuuint64_t gstride[1] = {(cuuint64_t)row_bytes};
    cuuint32_t box[2] = {(cuuint32_t)(row_bytes / element), (cuuint32_t)max(box_rows, 1)};
    cuuint32_t estr[2] = {1, 1};
    g_map_encodings.fetch_add(1, std::memory_order_relaxed);
    return fn(m, type, 2, const_cast<void *>(base), gdim, gstride, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, box_rows > 0 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
              CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The maps of a plane set, kept together: a serving loop calls with the same planes every step, layer after layer, and a
// call that encodes its ten maps takes the host 8.6 us where one that finds them takes 6.9.  What a map depends on is the key, compared in
// full.  At most MAX_PLANE_SETS sets (1.6 KB each, 7 MB) are kept, more than the layers of several models; past that the table begins anew, so
// that planes long gone make room.  (Ten look-ups of single maps took 7.4 us, and a table of 512 sets of four of them encoded
// 2461 of 3000 maps again in a second round over 300 layers.)
struct PlaneSetKey {
    const uint8_t *base[10];             // the planes in the order of S1GatherParams; those that no map is of are null
    int32_t dev, H, ps, num_pages, num_slots, nbi, nb, by_row;
    bool operator==(const PlaneSetKey &o) const { return memcmp(this, &o, sizeof(*this)) == 0; }
};
static_assert(sizeof(PlaneSetKey) == 10 * 8 + 8 * 4, "compared and hashed as bytes: no padding");
struct PlaneSetHash {
    size_t operator()(const PlaneSetKey &k) const {
        uint64_t w[sizeof(k) / 8], h = 0;
        memcpy(w, &k, sizeof(k));
        for (uint64_t x : w) { h = (h ^ x) * 0x9E3779B97F4A7C15ull; h ^= h >> 29; }
        return (size_t)h;
    }
};
struct PlaneSetMaps { CUtensorMap page_k, page_v, rows[10]; };
constexpr size_t MAX_PLANE_SETS = 4096;

int set_plane_maps(S1Params &p, CUtensorMap *rows) {
    if (rows == nullptr && p.H < 4) return 0;
    const uint8_t *base[10] = {p.k_base, p.v_main, p.v_scale, p.v_zp, p.k_scale, p.k_zp, p.k_ms, p.k_mc, p.k_obmp, p.k_oval};
    const int planes = rows == nullptr ? 2 : (p.k_out > 0 ? 10 : 6);
    PlaneSetKey key;
    memset(&key, 0, sizeof(key));
    for (int i = 0; i < planes; ++i) key.base[i] = base[i];
    if (int rc = current_device(&key.dev)) return rc;
    key.H = p.H; key.ps = p.ps; key.num_pages = p.num_pages;
    if (rows != nullptr) { key.by_row = 1; key.num_slots = p.num_slots; key.nbi = planes == 10 ? p.nbi : 0; key.nb = planes == 10 ? p.nb : 0; }
    typedef std::unordered_map<PlaneSetKey, PlaneSetMaps, PlaneSetHash> Table;
    static std::mutex mu;
    alignas(Table) static unsigned char room[sizeof(Table)];
    static Table &table = *new (room) Table;                             // never torn down under a thread that still decodes at exit
    auto hand_out = [&](const PlaneSetMaps &m) {
        if (p.H >= 4) { p.tmap_k = m.page_k; p.tmap_v = m.page_v; }
        if (rows != nullptr) memcpy(rows, m.rows, planes * sizeof(CUtensorMap));
    };
    {
        std::lock_guard<std::mutex> g(mu);
        const auto it = table.find(key);
        if (it != table.end()) { hand_out(it->second); return 0; }
    }
    PlaneSetMaps m;
    memset(&m, 0, sizeof(m));
    bool ok = true;
    if (p.H >= 4) {                                                      // a page is whole 1 KB swizzle atoms
        const int64_t bytes = (int64_t)p.num_pages * p.rows_per_page * 128;
        ok = encode_map(&m.page_k, p.k_base, bytes, 128, p.rows_per_page) && encode_map(&m.page_v, p.v_main, bytes, 128, p.rows_per_page);
    }
    if (rows != nullptr) {
        const int page = p.ps * p.H, slot = 128 * p.H, page_split = gather_page_split(p.GS * p.ppg), slot_split = gather_slot_split(p.H);
        const int bytes[10] = {32 * page, 32 * page, 4 * page, 8 * page, slot, 2 * slot, 2 * slot, 2 * slot, p.nbi * slot, p.nb * slot};
        for (int i = p.H == 4 ? 2 : 0; ok && i < planes; ++i) {
            const int row = bytes[i] / (i < 4 ? page_split : slot_split);
            if (i == 8 && row > GATHER_ROW_MAX) continue;                // copied slot by slot
            ok = encode_map(&m.rows[i], base[i], (int64_t)bytes[i] * (i < 4 ? p.num_pages : p.num_slots), row, 0);
        }
    }
    if (!ok) return fail(OMMX_E_CUDA, "stage 1: the tensor maps of the planes could not be encoded");
    hand_out(m);
    try {
        std::lock_guard<std::mutex> g(mu);
        if (table.size() >= MAX_PLANE_SETS) table.clear();
        table.emplace(key, m);
    } catch (const std::bad_alloc &) {}                                  // encoded again at the next call
    return 0;
}

static size_t stage1_smem(const S1Params &p) { return stage1_smem(p.nstages, p.stage_bytes, p.GS, p.ppg); }

// Never launched: a CTA of it takes a whole SM, as those of every form of stage 1 do, so as many clusters of it run at once, and
// the question loads no form that the process may never launch.
__global__ void whole_sm_kernel() {}
static int clusters_at_once(int cluster, int *n) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cluster);
    cfg.blockDim = dim3(WarpLayout<8, false>::THREADS);
    cfg.dynamicSmemBytes = SMEM_LIMIT;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    OMMX_CUDA_TRY(cudaFuncSetAttribute(whole_sm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_LIMIT));
    OMMX_CUDA_TRY(cudaOccupancyMaxActiveClusters(n, whole_sm_kernel, &cfg));
    return 0;
}
// The current device, asked once; where it does not say how many clusters of a size it runs, none are launched
static int current_chip(Chip *chip) {
    static std::atomic<uint64_t> known[MAX_DEVICES];   // 16 bits each: SMs, clusters of 2, 4 and 8
    int dev = 0;
    if (int rc = current_device(&dev)) return rc;
    uint64_t word = known[dev].load(std::memory_order_acquire);
    if (word == 0) {
        word = (uint64_t)(sm_count_of(dev) & 0xFFFF);
        for (int i = 0; i < 3; ++i) {
            int n = 0;
            if (clusters_at_once(2 << i, &n) != 0) { (void)cudaGetLastError(); n = 0; }
            word |= (uint64_t)(n & 0xFFFF) << (16 * (i + 1));
        }
        known[dev].store(word, std::memory_order_release);
    }
    *chip = Chip{(int)(word & 0xFFFF), {(int)(word >> 16 & 0xFFFF), (int)(word >> 32 & 0xFFFF), (int)(word >> 48)}};
    return 0;
}

static int stage1_launch(const ommx_decode_args *a, Stage1Grid *grid) {
    Chip chip;
    if (int rc = current_chip(&chip)) return rc;
    *grid = stage1_grid(a->batch, a->num_kv_splits, a->max_seq_len, chip);
    return 0;
}

}  // namespace ommx
#include "ommx_decode_tc.cuh"
namespace ommx {

// Which stage-1 kernel serves a call.  The register-operand kernel (decode_stage1_kernel) is the default: on B200 it
// is the faster of the two (37 us against 98 us for 64K tokens x 8 heads).  OMMX_B200_STAGE1=tc selects the tensor-core
// kernel (decode_stage1_tc_kernel) where its shared-memory plan fits - 4 or 8 local kv heads with GQA <= 4, fewer
// heads at any GQA <= 8 - and no differential-timing knob is set; it produces the same results within the path's
// tolerance and is kept for further work on its pipeline.  The variable is read once per call (`tc` below).
static bool tensor_core_stage1() {
    const char *e = getenv("OMMX_B200_STAGE1");
    return e && !strcmp(e, "tc");
}
// Its shared memory for this call (when it is asked for), or 0 where the default kernel serves
static size_t tensor_core_plan(const ommx_decode_args *a, const S1Params &p, TcParams *T) {
    if (p.abl != 0 || p.gqa > 8 || p.idx7) return 0;
    T->s = p;
    T->s.GS = 1;
    T->s.stage_bytes = p.gb_bytes;
    const int per_max = ((a->max_seq_len + a->num_kv_splits - 1) / a->num_kv_splits + 31) / 32;   // groups of the longest split
    const size_t smem = tc_layout(*T, p.gqa <= 4 ? 4 : 8, per_max + 1);
    return smem <= SMEM_LIMIT ? smem : 0;
}

static int fill_stage1(const ommx_decode_args *a, S1Params &p) {
    const ommx_kv_planes &pl = a->planes;
    p.q = (const __nv_bfloat16 *)a->q; p.q_sb = a->q_stride_b; p.q_sh = a->q_stride_h;
    p.B = a->batch; p.Hq = a->n_q_heads; p.H = pl.n_kv_heads; p.gqa = a->n_q_heads / pl.n_kv_heads;
    p.q_vec_ok = (((uintptr_t)a->q & 15) == 0 && a->q_stride_b % 8 == 0 && a->q_stride_h % 8 == 0) ? 1 : 0;
    p.k_base = (const uint8_t *)pl.k_base; p.v_main = (const uint8_t *)pl.v_main;
    p.v_scale = (const uint8_t *)pl.v_scale; p.v_zp = (const uint8_t *)pl.v_zp;
    p.k_scale = (const uint8_t *)pl.k_scale; p.k_zp = (const uint8_t *)pl.k_zp;
    p.k_ms = (const uint8_t *)pl.k_mapscale; p.k_mc = (const uint8_t *)pl.k_mapcenter;
    p.k_obmp = (const uint8_t *)pl.k_obmp; p.k_oval = (const uint8_t *)pl.k_oval;
    p.ps = pl.page_size; p.ppg = 32 / pl.page_size; p.num_pages = pl.num_pages; p.num_slots = pl.num_group_slots;
    p.k_out = pl.outliers_per_vector; p.nb = (pl.outliers_per_vector + 1) / 2;
    p.idx7 = (pl.outlier_index == OMMX_OIDX_RELIDX7 && pl.outliers_per_vector > 0) ? 1 : 0;
    p.nbi = p.idx7 ? (7 * pl.outliers_per_vector + 7) / 8 : 4;
    p.use_map = (pl.kv_outlier_map && pl.outliers_per_vector > 0) ? 1 : 0;
    p.b_seq_len = a->b_seq_len; p.r2t = a->req_to_token; p.r2g = a->req_to_group; p.tbl64 = a->table_is_int64;
    p.r2t_sb = a->r2t_stride_b; p.r2g_sb = a->r2g_stride_b;
    p.al = a->attn_logits; p.al_sb = a->al_stride_b; p.al_sh = a->al_stride_h; p.al_ss = a->al_stride_s;
    p.S = a->num_kv_splits; p.seg_group_base = a->seg_group_base;
    p.sm_scale = a->sm_scale; p.logit_cap = a->logit_cap; p.status = a->status;
    const int H = p.H;
    p.GS = NCW / H;
    p.o_vm = H * 1024; p.o_vs = H * 2048; p.o_vz = p.o_vs + H * 128; p.o_ks = p.o_vz + H * 256;
    p.o_kz = p.o_ks + H * 128; p.o_ms = p.o_kz + H * 256; p.o_mc = p.o_ms + H * 256; p.o_bm = p.o_mc + H * 256;
    p.o_ov = (p.o_bm + H * 128 * p.nbi + 15) / 16 * 16;
    p.gb_bytes = p.o_ov + H * 128 * (p.nb > 0 ? p.nb : 0);
    // swizzled tensor-map staging of the two code planes when a page is whole 1 KB swizzle atoms and
    // the 1 KB rounding of the group block still fits shared memory (4 or 8 local kv heads); set_plane_maps fills in the maps
    const int64_t page_bytes = (int64_t)p.ps * H * 32;
    p.swz = 0;
    p.rows_per_page = (int32_t)(page_bytes / 128);
    memset(&p.tmap_k, 0, sizeof(CUtensorMap));
    memset(&p.tmap_v, 0, sizeof(CUtensorMap));
    if (H >= 4) p.swz = 0x70u;                                           // a page is whole 1 KB swizzle atoms
    const int round_to = p.swz ? 1024 : 128;
    p.gb_bytes = (p.gb_bytes + round_to - 1) / round_to * round_to;
    p.stage_bytes = (p.GS * p.gb_bytes + 1023) / 1024 * 1024;
    p.abl = a->abl_flags;
    return 0;
}

// Stage 1's launch, without CTAs where it makes equal splits per sequence (the tensor-core kernel): stage 2 works out the same
// workspace slots from it
static int shared_grid(const ommx_decode_args *a, bool tc, Stage1Grid *grid) {
    if (tc) {
        S1Params p;
        TcParams T;
        if (int rc = fill_stage1(a, p)) return rc;
        if (int rc = set_plane_maps(p, nullptr)) return rc;              // what stage 1 refuses, stage 2 by itself refuses too
        if (tensor_core_plan(a, p, &T)) { *grid = Stage1Grid{0, 0, 1, 0}; return 0; }
    }
    return stage1_launch(a, grid);
}

static int launch_stage1(const ommx_decode_args *a, cudaStream_t st, bool tc) {
    if (a->max_seq_len <= 0) return 0;                                   // tail-only decode
    S1Params p;
    if (int rc = fill_stage1(a, p)) return rc;
    if (tc) {
        if (int rc = set_plane_maps(p, nullptr)) return rc;
        TcParams T;
        if (const size_t tsmem = tensor_core_plan(a, p, &T)) {
            dim3 tgrid(a->num_kv_splits, a->batch);
            if (p.gqa <= 4) return p.H == 8 ? launch_tc<4, true>(T, tgrid, tsmem, st) : launch_tc<4, false>(T, tgrid, tsmem, st);
            return p.H == 8 ? launch_tc<8, true>(T, tgrid, tsmem, st) : launch_tc<8, false>(T, tgrid, tsmem, st);
        }
    }
    // deepest ring that fits the 227 KB a CTA may use
    p.nstages = MAX_STAGES;
    while (p.nstages > 2 && stage1_smem(p) > SMEM_LIMIT) --p.nstages;
    const size_t smem = stage1_smem(p);
    if (smem > SMEM_LIMIT) return fail(OMMX_E_UNSUPPORTED, "stage 1 planes of one group do not fit shared memory");
    if (int rc = stage1_launch(a, &p.grid)) return rc;
    switch (p.H) {
        case 8: return launch_stage1_h8(p, smem, st);
        case 4: return launch_stage1_h4(p, smem, st);
        case 2: return launch_stage1_h2(p, smem, st);
        default: return launch_stage1_h1(p, smem, st);
    }
}

// `after_stage1`: the previous kernel in the stream is this call's own stage 1, so stage 2 may be
// launched as its programmatic dependent.
static int launch_stage2(const ommx_decode_args *a, cudaStream_t st, bool tc, bool after_stage1) {
    const ommx_kv_planes &pl = a->planes;
    S2Params p;
    p.q = (const __nv_bfloat16 *)a->q; p.q_sb = a->q_stride_b; p.q_sh = a->q_stride_h;
    p.Hq = a->n_q_heads; p.gqa = a->n_q_heads / pl.n_kv_heads; p.D = pl.head_dim;
    p.k_tail = (const __nv_bfloat16 *)a->k_tail; p.v_tail = (const __nv_bfloat16 *)a->v_tail;
    p.t_sb = a->tail_stride_b; p.t_st = a->tail_stride_t; p.t_sh = a->tail_stride_h;
    p.b_tail_len = a->max_tail_len > 0 ? a->b_tail_len : nullptr; p.b_seq_len = a->b_seq_len;
    p.max_tail = a->max_tail_len;
    p.v_vec_ok = (((uintptr_t)a->v_tail & 7) == 0 && a->tail_stride_b % 4 == 0 && a->tail_stride_t % 4 == 0 && a->tail_stride_h % 4 == 0) ? 1 : 0;
    p.al = a->attn_logits; p.al_sb = a->al_stride_b; p.al_sh = a->al_stride_h; p.al_ss = a->al_stride_s;
    p.S = a->max_seq_len > 0 ? a->num_kv_splits : 0;
    p.B = a->batch; p.grid = Stage1Grid{0, 0, 1, 0};
    if (p.S > 0)
        if (int rc = shared_grid(a, tc, &p.grid)) return rc;
    p.by = share_divisors(p.grid, max(p.S, 1));
    p.o = a->o; p.o_bf16 = (a->o_dtype == OMMX_DT_BF16); p.o_sb = a->o_stride_b; p.o_sh = a->o_stride_h;
    p.lse = a->lse; p.lse_sb = a->lse_stride_b;
    p.sm_scale = a->sm_scale; p.logit_cap = a->logit_cap;
    p.g_world = 0; p.g_rank = 0; p.g_recv = nullptr; p.g_out = nullptr; p.g_state = nullptr; p.status = a->status;
    if (a->gather) {
        const ommx_head_gather *g = a->gather;
        if (g->world < 2 || g->world > 32 || g->rank < 0 || g->rank >= g->world || !g->recv || !g->out || !g->state)
            return fail(OMMX_E_ARG, "head gather: world must be 2..32, rank inside it, and recv / out / state set");
        p.g_world = g->world; p.g_rank = g->rank; p.g_recv = g->recv; p.g_out = g->out; p.g_state = g->state;
    }
    int warps;
    Stage2Kernel kernel;
    {
        // Stage 1 runs with the largest shared-memory carve-out; asking for the same split here spares the SMs a
        // reconfiguration between the two kernels of every layer.
        static const Stage2Kernel all[] = {decode_stage2_kernel<16, 1, false>, decode_stage2_kernel<8, 2, false>, decode_stage2_kernel<4, 4, false>,
                                           decode_stage2_kernel<4, 7, false>, decode_stage2_kernel<16, 1, true>, decode_stage2_kernel<8, 2, true>,
                                           decode_stage2_kernel<4, 4, true>, decode_stage2_kernel<4, 7, true>};
        static std::atomic<int> carve_set[MAX_DEVICES];
        int dev = 0;
        if (int rc = current_device(&dev)) return rc;
        if (carve_set[dev].load(std::memory_order_acquire) == 0) {
            for (Stage2Kernel k : all)
                OMMX_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared));
            carve_set[dev].store(1, std::memory_order_release);
        }
        // the largest CTAs of which all rows still run at once
        const long long rows = (long long)a->n_q_heads * a->batch, sms = sm_count_of(dev);
        const int size = rows <= sms ? 0 : (rows <= 2 * sms ? 1 : (rows <= 4 * sms ? 2 : 3));
        kernel = all[size + (p.grid.cluster > 1 ? 4 : 0)];
        warps = size == 0 ? 16 : (size == 1 ? 8 : 4);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a->n_q_heads, a->batch);
    cfg.blockDim = dim3(32 * warps);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;   // overlap this kernel's prologue with stage 1's tail
    cfg.attrs = attr;
    cfg.numAttrs = (after_stage1 && a->max_seq_len > 0) ? 1 : 0;
    OMMX_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, p));
    count_launch();
    return 0;
}

}  // namespace ommx

extern "C" int ommx_b200_min_num_kv_splits(int32_t max_seq_len, int32_t page_size) {
    using namespace ommx;
    if (max_seq_len <= 0) return 1;
    int ppg = page_size > 0 && page_size <= 32 ? 32 / page_size : 1;
    int max_groups = MAX_SPLIT_GROUPS;
    if (max_groups * ppg > MAX_SPLIT_PAGES) max_groups = MAX_SPLIT_PAGES / ppg;
    const int groups = (max_seq_len + 31) / 32;
    return (groups + max_groups - 1) / max_groups;
}

extern "C" int ommx_b200_auto_num_kv_splits(int32_t max_seq_len, int32_t batch, int32_t n_kv_heads) {
    (void)n_kv_heads;                       // one CTA serves all local kv heads of its token range
    const int sm_count = ommx::sm_count();
    // For sequences of one length in equal splits: one CTA runs per SM, so a launch takes (waves of CTAs) x (groups per CTA +
    // what a CTA costs before and after its steady state, about three groups' worth).  Pick the split count that minimises it:
    // 147 or 148 at batch 1, and e.g. 18 rather than 19 at batch 8, where 152 CTAs would leave a second wave of four.  Ties go to
    // fewer splits (less for stage 2 to combine).  A ragged batch is shared out more evenly with more slots (share_plan_of).
    const int groups = max(1, (max_seq_len + 31) / 32);
    const int b = max(1, batch);
    const int s_min = ommx_b200_min_num_kv_splits(max_seq_len, 16);
    const int s_max = max(s_min, min(groups, (4 * sm_count) / b + 1));
    int best = s_min;
    long long best_cost = -1;
    for (int s = s_min; s <= s_max; ++s) {
        const long long waves = ((long long)b * s + sm_count - 1) / sm_count;
        const long long cost = waves * ((groups + s - 1) / s + 3);
        if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = s; }
    }
    return max(1, best);
}

extern "C" int ommx_b200_host_launch_plan(const int32_t *b_seq_len, int32_t batch, int32_t num_kv_splits, int32_t max_seq_len, int32_t sm_count,
                                          const int32_t *clusters_at_once, ommx_launch_plan *out) {
    using namespace ommx;
    if (!b_seq_len || !out || batch < 1 || num_kv_splits < 1 || sm_count < 0)
        return fail(OMMX_E_ARG, "host_launch_plan: batch=%d num_kv_splits=%d sm_count=%d", batch, num_kv_splits, sm_count);
    Chip chip = chip_of(sm_count);
    if (sm_count == 0)
        if (int rc = current_chip(&chip)) return rc;
    if (sm_count > 0 && clusters_at_once)
        for (int i = 0; i < 3; ++i) {
            if (clusters_at_once[i] < 0 || clusters_at_once[i] > sm_count >> (i + 1))
                return fail(OMMX_E_ARG, "host_launch_plan: %d clusters of %d CTAs on %d SMs", clusters_at_once[i], 2 << i, sm_count);
            chip.clusters[i] = clusters_at_once[i];
        }
    int total = 0, longest = 0;
    for (int i = 0; i < batch; ++i) {
        total += groups_of(b_seq_len[i]);
        longest = max(longest, groups_of(b_seq_len[i]));
    }
    const Stage1Grid grid = stage1_grid(batch, num_kv_splits, max_seq_len, chip);
    const SharePlan plan = share_plan_of(total, longest, batch, num_kv_splits, grid, share_divisors(grid, num_kv_splits));
    *out = ommx_launch_plan{grid.ncta, grid.cluster, plan.shares, plan.ctas, plan.per};
    return MAX_PIECES;
}
extern "C" int ommx_b200_host_share_plan(const int32_t *b_seq_len, int32_t batch, int32_t num_kv_splits, int32_t max_seq_len, int32_t sm_count,
                                         int32_t *ctas, int32_t *groups_per_cta) {
    using namespace ommx;
    if (!ctas || !groups_per_cta || sm_count < 1) return fail(OMMX_E_ARG, "host_share_plan: null output or sm_count=%d", sm_count);
    ommx_launch_plan plan;
    const int limit = ommx_b200_host_launch_plan(b_seq_len, batch, num_kv_splits, max_seq_len, sm_count, nullptr, &plan);
    if (limit < 0) return limit;
    *ctas = plan.shares;
    *groups_per_cta = plan.groups_per_share;
    return limit;
}

extern "C" int64_t ommx_b200_tensor_map_encodings(void) { return (int64_t)ommx::g_map_encodings.load(); }

extern "C" int ommx_b200_decode_stage1(const ommx_decode_args *a, void *stream) {
    int rc = ommx::validate_decode(a);
    if (rc) return rc;
    return ommx::launch_stage1(a, (cudaStream_t)stream, ommx::tensor_core_stage1());
}
extern "C" int ommx_b200_decode_stage2(const ommx_decode_args *a, void *stream) {
    int rc = ommx::validate_decode(a);
    if (rc) return rc;
    return ommx::launch_stage2(a, (cudaStream_t)stream, ommx::tensor_core_stage1(), false);
}
extern "C" int ommx_b200_decode(const ommx_decode_args *a, void *stream) {
    int rc = ommx::validate_decode(a);
    if (rc) return rc;
    const bool tc = ommx::tensor_core_stage1();
    rc = ommx::launch_stage1(a, (cudaStream_t)stream, tc);
    if (rc) return rc;
    return ommx::launch_stage2(a, (cudaStream_t)stream, tc, true);
}

// -------------------------------------------------------------------------------------------------
// Decode with the split workspace owned by the library.
//
// Some hosts that embed this library may not allocate device memory at all on their serving path:
// a runtime whose allocator has been frozen after start-up (every later cudaMalloc would fragment or
// overrun a pool sized to the last megabyte), or a plug-in that is handed tensors but no allocator.
// ommx_b200_decode needs a workspace for the per-split partial results; this entry point takes it
// from a fixed array inside the library image instead, so the caller passes only inputs and outputs.
// The array is part of the module: every GPU that loads the library holds its 8 MiB until exit.
constexpr size_t STATIC_WS_FLOATS = (size_t)2 << 20;                      // 2 Mi floats = 8 MiB
static __device__ __align__(256) float g_static_ws[STATIC_WS_FLOATS];

// In host code the name g_static_ws is only a handle, not a device address; the address each
// device gave the array is asked for once per device, with that device current, and kept.
static int static_ws_address(float **out) {
    static std::atomic<float *> cache[64];
    int dev = -1;
    OMMX_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return ommx::fail(OMMX_E_UNSUPPORTED, "decode_static_ws: device ordinal %d", dev);
    float *ptr = cache[dev].load(std::memory_order_acquire);
    if (ptr == nullptr) {
        void *sym = nullptr;
        OMMX_CUDA_TRY(cudaGetSymbolAddress(&sym, g_static_ws));
        if (sym == nullptr) return ommx::fail(OMMX_E_CUDA, "decode_static_ws: the workspace symbol has no address on device %d", dev);
        ptr = static_cast<float *>(sym);
        cache[dev].store(ptr, std::memory_order_release);
    }
    *out = ptr;
    return 0;
}

extern "C" int ommx_b200_decode_static_ws(const ommx_decode_args *a, void *stream) {
    using namespace ommx;
    if (!a) return fail(OMMX_E_ARG, "decode_static_ws: null args");
    if (a->batch <= 0 || a->n_q_heads <= 0 || a->num_kv_splits <= 0)
        return fail(OMMX_E_ARG, "decode_static_ws: batch=%d n_q_heads=%d num_kv_splits=%d", a->batch, a->n_q_heads, a->num_kv_splits);
    const size_t row = (size_t)HD + 1;
    const size_t need = (size_t)a->batch * a->n_q_heads * a->num_kv_splits * row;
    if (need > STATIC_WS_FLOATS)
        return fail(OMMX_E_ARG, "decode_static_ws: batch*n_q_heads*num_kv_splits*(head_dim+1) = %zu floats exceeds the "
                                "built-in workspace of %zu floats (8 MiB); use ommx_b200_decode with your own attn_logits",
                    need, (size_t)STATIC_WS_FLOATS);
    float *ws = nullptr;
    int rc = static_ws_address(&ws);
    if (rc) return rc;
    ommx_decode_args b = *a;
    b.attn_logits = ws;
    b.al_stride_s = (int64_t)row;
    b.al_stride_h = (int64_t)a->num_kv_splits * (int64_t)row;
    b.al_stride_b = (int64_t)a->n_q_heads * b.al_stride_h;
    rc = validate_decode(&b);
    if (rc) return rc;
    const bool tc = tensor_core_stage1();
    rc = launch_stage1(&b, (cudaStream_t)stream, tc);
    if (rc) return rc;
    return launch_stage2(&b, (cudaStream_t)stream, tc, true);
}

extern "C" int ommx_b200_merge_states(const float *o_parts, const float *lse_parts, const int32_t *valid_lens,
                                      int32_t P, int32_t R, int32_t D, float *o, float *lse, void *stream) {
    using namespace ommx;
    if (!o_parts || !lse_parts || !o || !lse) return fail(OMMX_E_ARG, "merge: null pointer");
    if (P < 0 || R < 0 || D <= 0) return fail(OMMX_E_ARG, "merge: P=%d R=%d D=%d", P, R, D);
    if (R == 0) return 0;
    merge_states_kernel<<<R, 128, 0, (cudaStream_t)stream>>>(o_parts, lse_parts, valid_lens, P, R, D, o, lse);
    OMMX_CUDA_TRY(cudaGetLastError());
    count_launch();
    return 0;
}

// Stage 1 of the paged decode: the kernel, its launch, and what the tensor-core form (ommx_decode_tc.cuh) shares with it.  Each
// kv-head count is a translation unit of its own (ommx_stage1_h8.cu ...), so that they compile side by side.
#pragma once
#include "ommx_common.cuh"
#include <cuda.h>                       // CUtensorMap (types only; the encoder is looked up at run time)
#include <mutex>
#include <stdlib.h>
#include <string.h>
#include <type_traits>

namespace ommx {

constexpr int HD = 128;                 // head_dim this build serves
constexpr int NCW = 8;                  // (group, head) units in flight per CTA, one MMA warp each
// Two warp layouts.  Narrow (2, 4 or 8 local kv heads: 14 to 16 copies per ring stage): 15 decode warps + 1 producer warp,
// which also builds the last tile half once its copies are out.  Wide (1 local kv head: a stage is 8 groups, 28 copies; in the
// general form, which copies page by page and slot by slot, 112, and 56 with 2 heads): 16 decode warps + 4 producer warps, because
// one warp issues a copy only every ~60 cycles on an idle SM, three times that beside the other roles, and the issues of different
// warps overlap.  One producer keeps up with about 20 copies a stage: 8 x 32K, one head, four rows to a copy 31.8 us by one
// producer and 31.0 by four; 128K, two heads, 14 copies 28.2 and 28.6.
template <int H, bool GATHER> struct WarpLayout {
    static constexpr bool WIDE = H == 1 || (H == 2 && !GATHER);
    static constexpr int NDW = WIDE ? 16 : 15;            // decode warps (stateless sidecar builders, items dealt round-robin)
    static constexpr int NPW = WIDE ? 4 : 1;              // producer warps
    static constexpr int PRODUCER_WARP = NCW + NDW;       // the first of them
    static constexpr int THREADS = (NCW + NDW + NPW) * 32;
};
// Register budget per role (setmaxnreg, warpgroup granularity).  Only what the CTA was launched with
// can be moved around: 768 threads x 80 = 61440 = 256*128 (MMA) + 512*56 (decode + producer).  The
// launch refuses to run if the compiled kernel holds fewer registers than the roles ask for, because
// setmaxnreg.inc would then wait forever.
#define OMMX_REGS_MMA "128"
#define OMMX_REGS_DECODE "56"
#define OMMX_REGS_PRODUCER "24"
constexpr int REGS_MMA = 128, REGS_DECODE = 56, REGS_PRODUCER = 24;
constexpr int MAX_STAGES = 4;           // ring depth (3 when the planes of a stage are large)
constexpr int DT_STRIDE = 272;          // bytes per sidecar-tile row (256 data + 16 pad)
constexpr int ROW_KF = 32;              // K scale factors 2^(e + KF_BIAS) * 4^-slot, bf16, in code-fragment order
constexpr int ROW_VF = 33;              // V scale factors, fp16, fragment order (rows 33, 34: two copies)
constexpr int DT_ROWS = 35;             // rows 0..31: outlier deltas [token][channel in fragment order], bf16
constexpr int DT_BYTES = DT_ROWS * DT_STRIDE;
constexpr int MAX_SPLIT_GROUPS = 512;   // groups of the longest split that the entry points accept (16K tokens)
constexpr int MAX_SPLIT_PAGES = 1024;
constexpr int MAX_PIECES = 128;         // pieces of sequences one CTA can work on (32 bytes of shared memory each)
constexpr long long WAIT_LIMIT_CYCLES = 2000000000ll;   // about a second of SM clock: the wait has failed

// The launch: CTAs (one per SM at most) in clusters of `cluster`; rounds of CTAs (clusters) that B * S splits would take
struct Stage1Grid { int32_t ncta, waves, cluster, cluster_waves; };
// What it is made for: SMs, and how many clusters of 2, 4 and 8 CTAs of one SM each run at once
struct Chip { int sms, clusters[3]; };

// Division by what a launch knows beforehand: stage 1 prepares the reciprocals before it waits for the kernel ahead of it (three divisions
// between the lengths and the first copy were 0.8 us of every launch; from the host, among the parameters, 8 x 32K 136.7 -> 137.1),
// stage 2, of which they were a quarter of the instructions, gets them from the host.  Exact: with m = floor((2^32 - 1) / d) the product's upper half
// is the quotient or one less.
struct Divisor {
    uint32_t d, m;
    __host__ __device__ __forceinline__ int of(int n) const {        // n / d for n >= 0
        const uint32_t q = (uint32_t)(((uint64_t)(uint32_t)n * m) >> 32);
        return (int)(q + ((uint32_t)n - q * d >= d ? 1u : 0u));
    }
};
__host__ __device__ __forceinline__ Divisor divisor(int d) { return Divisor{(uint32_t)d, 0xFFFFFFFFu / (uint32_t)d}; }
struct ShareDivisors { Divisor ctas, shares, slots, slots1; };        // CTAs, clusters, S, S - 1
__host__ __device__ __forceinline__ ShareDivisors share_divisors(const Stage1Grid &g, int S) {
    return ShareDivisors{divisor(max(g.ncta, 1)), divisor(max(g.ncta / max(g.cluster, 1), 1)), divisor(S), divisor(max(S - 1, 1))};
}

struct S1Params {
    const __nv_bfloat16 *q;
    int64_t q_sb, q_sh;
    int32_t B, Hq, H, gqa, q_vec_ok;     // q_vec_ok: eight adjacent q elements may be fetched as one 16-byte word
    const uint8_t *k_base, *v_main, *v_scale, *v_zp, *k_scale, *k_zp, *k_ms, *k_mc, *k_obmp, *k_oval;
    int32_t ps, ppg, num_pages, num_slots, k_out, nb, use_map;
    int32_t nbi;                         // bytes of outlier index per channel: 4 (flat bitmask) or ceil(7k/8) (relidx7, idx7 = 1)
    int32_t idx7;
    const int32_t *b_seq_len;
    const void *r2t, *r2g;
    int32_t tbl64;
    int64_t r2t_sb, r2g_sb;
    float *al;
    int64_t al_sb, al_sh, al_ss;
    int32_t S, seg_group_base;
    Stage1Grid grid;
    float sm_scale, logit_cap;
    int32_t *status;
    int32_t abl;
    // shared-memory layout of one group block (bytes)
    int32_t GS, gb_bytes, stage_bytes, nstages;
    int32_t o_vm, o_vs, o_vz, o_ks, o_kz, o_ms, o_mc, o_bm, o_ov;
    // tensor maps of the two code planes as [bytes/128][128] uint8 with 128-byte swizzle
    uint32_t swz;                        // 0x70 when the maps are in use, else 0
    int32_t rows_per_page;               // 128-byte lines per page
    alignas(64) CUtensorMap tmap_k;
    alignas(64) CUtensorMap tmap_v;
};
// One to four kv heads, plain form: a stage holds several groups, so its copies are many and small, and issuing them is what a stage
// waits for (they go out one by one, ~30 instructions each).  Its planes are laid out for all its groups at once, so that one
// instruction fetches four pages or group slots (`tile::gather4`): 28, 14 and 16 copies at 1, 2 and 4 heads for 112, 56 and 28.  Both
// stages, before -> now: 128K x 2 heads 28.8 -> 28.1 us, 256K 46.1 -> 44.2; 8 x 32K x 1 head 33.9 -> 30.6, 512K 51.7 -> 44.3; 128K x 4
// heads 46.1 -> 43.5, 32K 19.5 (no change).  Rows of two heads lie as they come (conflicts: a token row is 64 bytes): by page with a
// swizzle they need 26 copies, 28.8 us.  Eight heads have a group to a stage and nothing to fold.
// These are the tensor maps of the planes as they are numbered below, a page or group slot to a row.
struct S1GatherParams : S1Params {
    CUtensorMap rows[10];
};
// the planes: 0 k_base, 1 v_main, 2 v_scale, 3 v_zp by page; 4 k_scale, 5 k_zp, 6 map scale, 7 map center, 8 outlier index, 9 outlier values by slot
constexpr int GATHER_ROW_MAX = 2048;     // bytes of a row: 256 elements of 8 bytes
__host__ __device__ constexpr int gather_slot_split(int heads) { return heads == 4 ? 2 : 1; }          // rows of a group slot
__host__ __device__ constexpr int gather_page_split(int stage_pages) { return stage_pages < 4 ? 2 : 1; }   // of a page (planes 2 and 3)

// One bulk copy of a stage: source plane, bytes, destination inside the stage, and which table entry
// (page id or group slot) selects the source block.
struct __align__(16) CopyDesc {
    const uint8_t *src;                  // plane base, or nullptr + kind for a tensor-map copy
    uint32_t unit, dst;
    int32_t tbase, tmul, gi, tok0;       // gi: group in stage (bits 0..7) | kind << 8
};                                       // kind 0 bulk copy, 1 k_base through tmap_k, 2 v_main through tmap_v, 3 + n four rows of plane n
// a stage holds at most 8 groups x (4 planes x 4 pages + 6 group planes) = 176 copies (1 kv head, 8-token pages)

// ---- PTX wrappers --------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait: returns false (and the caller raises OMMX_ST_TIMEOUT) instead of spinning forever.
// try_wait already parks the warp in hardware for a short while.  The limit is counted on the SM
// clock (cheap to read); nanosleep or the global timer in this loop would put their own latency
// on every producer/consumer hand-off.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, long long limit = WAIT_LIMIT_CYCLES) {
    long long t_end = 0;
#pragma unroll 1
    for (uint32_t i = 1; !mbar_try_wait(bar, parity); ++i) {
        if ((i & 63u) == 0) {
            const long long now = clock64();
            if (t_end == 0) t_end = now + limit;
            else if (now > t_end) return false;
        }
    }
    return true;
}
// ---- between the CTAs of a cluster: the address of a peer's shared memory, a release-arrive there, an acquire-wait here, a load ----
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t peer_smem(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_arrive_peer(uint32_t peer_bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(peer_bar) : "memory");
}
__device__ __forceinline__ bool mbar_wait_peers(uint32_t bar, uint32_t parity, long long limit) {
    const long long t_end = clock64() + limit;
    for (;;) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
        if (clock64() > t_end) return false;
    }
}
__device__ __forceinline__ float lds_peer(uint32_t peer_addr) {
    float x;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(peer_addr) : "memory");
    return x;
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                        uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// two 16x16 byte matrices (rows from lanes 0-15 and 16-31), transposed: r[2m], r[2m+1] = rows 4j..4j+3 of columns g and
// g + 8 of matrix m (lane = 4g + j)
__device__ __forceinline__ void ldsm_b8_trans_x2(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m16n16.x2.trans.shared.b8 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t addr, uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr) : "memory");
}
// transpose an 8x8 matrix of 16-bit elements held one row pair per lane (the accumulator layout)
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t x) {
    uint32_t r;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(x));
    return r;
}
__device__ __forceinline__ uint32_t pack_f16x2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ uint32_t pack_f16x2_sat(float lo, float hi) {       // clamped to the finite range
    uint32_t r;
    asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ uint32_t hmul2_bf16(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t hmul2_f16(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ uint32_t top_bit(uint32_t x) {                      // index of the highest set bit
    uint32_t r;
    asm("bfind.u32 %0, %1;" : "=r"(r) : "r"(x));
    return r;
}
__device__ __forceinline__ void sub_if_bit(float &x, uint32_t word, uint32_t bit, float y) {   // one logic instruction and a predicated add
    asm("{\n .reg .pred q;\n .reg .b32 t;\n and.b32 t, %1, %2;\n setp.ne.u32 q, t, 0;\n @q sub.f32 %0, %0, %3;\n}\n" : "+f"(x) : "r"(word), "r"(bit), "f"(y));
}
__device__ __forceinline__ void sts_u16x2(uint32_t a0, uint32_t a1, uint32_t x) {              // the halves of x to two places
    asm volatile("{\n .reg .b16 l, h;\n mov.b32 {l, h}, %2;\n st.shared.b16 [%0], l;\n st.shared.b16 [%1], h;\n}\n" ::"r"(a0), "r"(a1), "r"(x) : "memory");
}

// The 2-bit code planes are staged with the TMA's 128-byte swizzle (16-byte chunk index XOR line
// index mod 8) when a page is a whole number of 1 KB swizzle atoms: a head's 32-byte code row then
// lands in a different bank window on each token row instead of the same one.  `o` is the linear byte
// offset inside a 1 KB aligned region; swz is 0x70 (swizzled) or 0 (plain bulk copies).
__device__ __forceinline__ uint32_t swz128(uint32_t o, uint32_t swz) { return o ^ ((o >> 3) & swz); }

__device__ __forceinline__ void tma_2d_g2s(uint32_t dst, const CUtensorMap *map, int32_t x, int32_t y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}

// four rows of a plane, one after the other in shared memory
__device__ __forceinline__ void tma_rows_g2s(uint32_t dst, const CUtensorMap *map, const int4 &row, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];"
                 ::"r"(dst), "l"(map), "r"(0), "r"(row.x), "r"(row.y), "r"(row.z), "r"(row.w), "r"(bar) : "memory");
}

__device__ __forceinline__ int64_t load_index(const void *tbl, int is64, int64_t i) {
    return is64 ? reinterpret_cast<const int64_t *>(tbl)[i] : (int64_t) reinterpret_cast<const int32_t *>(tbl)[i];
}

// =================================================================================================
// Stage 1
// =================================================================================================
// Ablation bits (differential timing only, they break parity; mirror of the reference's
// OMMX_ABL_* knobs, paged_decode.py:3267-3279): 1 = skip the outlier splice, 2 = skip V dequant
// and P.V, 4 = skip the K code dequant and its MMAs.
constexpr int ABL_NO_OUTLIER = 1, ABL_NO_V = 2, ABL_NO_K = 4, ABL_NO_COMPUTE = 8;   // 8: stream the planes only
// 16 (tests of the give-up path only): waits give up after about 2 ms and the producer announces the bytes of its
// second ring fill without issuing the copies, so that every role runs out of patience and leaves through the epilogue
constexpr int ABL_TEST_STALL = 16;
constexpr long long TEST_WAIT_LIMIT_CYCLES = 4000000ll;

// V scale factors are fp16, 2^(e + FBIAS): exponents below -18 give 0 (such a scale step is under 2^-18 and the term it multiplies
// is dropped), exponents above 11 are clamped and reported.  K scale factors are bf16, 2^(e + KF_BIAS), clamped alike.
constexpr int FBIAS = 4;
constexpr int KF_BIAS = 70;
constexpr int E_TOP = 11 + 128;
constexpr float LAG = 0.68f;            // how far a logit may be ahead of the maximum that P is taken against: e^LAG * 2^(11 + FBIAS) < 65504
constexpr float KF_UNDO = 9223372036854775808.f;      // 2^(133 - KF_BIAS): a code field in place is code * 4^slot * 2^-133
__host__ __device__ constexpr uint32_t half2_const(int lo, int hi) { return ((uint32_t)lo & 0xFFFFu) | ((uint32_t)hi << 16); }
// the FP4 levels of four outliers (16 bits of the nibble stream) as the upper bytes of their fp16 values; the lower
// bytes are zero.  A nibble is the byte selector of the magnitude table; its sign bit, which as a selector bit replicates
// a byte's sign, turns 0x80 into 0xFF in a second lookup.
__device__ __forceinline__ uint32_t fp4_levels_hi(uint32_t nibbles) {
    const uint32_t mag = __byte_perm(0x3E3C3800u, 0x46444240u, nibbles & 0x7777u);
    uint32_t sgn;
    asm("prmt.b32 %0, %1, %1, %2;" : "=r"(sgn) : "r"(0x80808080u), "r"(nibbles));
    return mag | ((sgn << 7) & 0x80808080u);
}
__device__ __forceinline__ uint32_t f16_bits_sat(float x) {
    uint16_t r;
    asm("cvt.rn.satfinite.f16.f32 %0, %1;" : "=h"(r) : "f"(x));
    return (uint32_t)r;
}
// field i (0..7) of the lower and upper 8 codes of a 32-bit code word, as two bf16 subnormals code * 4^slot * 2^-133 with
// slot = i % 4 (7 mantissa bits and the lowest exponent bit: linear up to there): no arithmetic beyond the AND
__device__ __forceinline__ uint32_t code_pair_bf16(uint32_t w, int i) { return (i < 4 ? w : w >> 8) & (0x00030003u << (2 * (i & 3))); }
// Bit planes of the 2-bit codes of 64 channels x 32 tokens, the codes of a channel pair to a lane: w[0], w[1] are the low and the
// high code bit of its first channel, w[2], w[3] of its second, token = bit.  `addr` is the lane's row for the ldmatrix below:
// the 16 bytes of token 8 (lane / 4 % 4) + 4 (lane / 16) + lane % 4.  Lane 4g + j gets byte column g (j < 2) or g + 8, channels
// 2 (j & 1) and one more of it.
__device__ __forceinline__ void code_bit_planes(uint32_t addr, int lane, uint32_t (&w)[4]) {
    const bool right = lane & 2, odd = lane & 1;
    uint32_t r[4];
    ldsm_b8_trans_x2(addr, r);                               // r[2m + c]: tokens of quad j of matrix m, column g + 8c
    uint32_t own[2], oth[2];                                 // this lane's column: quads j and j ^ 2
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        own[m] = right ? r[2 * m + 1] : r[2 * m];
        oth[m] = __shfl_xor_sync(0xFFFFFFFFu, right ? r[2 * m] : r[2 * m + 1], 2);
    }
    // nibbles: both matrices' tokens side by side, the lower or upper channel pair; the other pair goes to the neighbour
    const uint32_t LO = 0x0F0F0F0Fu;
    const uint32_t a = (own[0] & LO) | ((own[1] << 4) & ~LO), b = ((own[0] >> 4) & LO) | (own[1] & ~LO);
    const uint32_t c = (oth[0] & LO) | ((oth[1] << 4) & ~LO), d = ((oth[0] >> 4) & LO) | (oth[1] & ~LO);
    const uint32_t q0 = odd ? b : a, q2 = odd ? d : c;                                            // quads j, j ^ 2
    const uint32_t q1 = __shfl_xor_sync(0xFFFFFFFFu, odd ? a : b, 1), q3 = __shfl_xor_sync(0xFFFFFFFFu, odd ? c : d, 1);   // j ^ 1, j ^ 3
    // quads in order in the bytes, the token inside its quad to the register
    const uint32_t s01 = odd ? 0x1504u : 0x5140u, s23 = odd ? 0x3726u : 0x7362u;
    const uint32_t e01 = __byte_perm(q0, q1, s01), e23 = __byte_perm(q0, q1, s23), f01 = __byte_perm(q2, q3, s01), f23 = __byte_perm(q2, q3, s23);
    const uint32_t h0 = right ? 0x1054u : 0x5410u, h1 = right ? 0x3276u : 0x7632u;
    const uint32_t a0 = __byte_perm(e01, f01, h0), a1 = __byte_perm(e01, f01, h1), a2 = __byte_perm(e23, f23, h0), a3 = __byte_perm(e23, f23, h1);
    // a_k, nibble n, bit i -> w_i, nibble n, bit k
    const uint32_t P = 0x33333333u, Q = 0x55555555u;
    const uint32_t b0 = (a0 & P) | ((a2 << 2) & ~P), b2 = ((a0 >> 2) & P) | (a2 & ~P);
    const uint32_t b1 = (a1 & P) | ((a3 << 2) & ~P), b3 = ((a1 >> 2) & P) | (a3 & ~P);
    w[0] = (b0 & Q) | ((b1 << 1) & ~Q); w[1] = ((b0 >> 1) & Q) | (b1 & ~Q);
    w[2] = (b2 & Q) | ((b3 << 1) & ~Q); w[3] = ((b2 >> 1) & Q) | (b3 & ~Q);
}

// stage index and phase parity of ring use number `it` (ring depth ns: 4 unless the planes are large)
__device__ __forceinline__ int ring_slot(int it, int ns) { return ns == 4 ? (it & 3) : it % ns; }
__device__ __forceinline__ uint32_t ring_phase(int it, int ns) { return (uint32_t)(ns == 4 ? (it >> 2) : it / ns) & 1u; }

// the bits of a pair's position stream (two streams of `bytes` bytes, k positions each) that only positions past 31 set
struct PositionBits { uint32_t word[8]; };
__host__ __device__ constexpr PositionBits past_31_bits(int k, int bytes) {
    PositionBits m = {};
    for (int i = 0; i < 2 * k; ++i)
        for (int b = 5; b < 7; ++b) {
            const int at = (i < k ? 0 : 8 * bytes) + 7 * (i % k) + b;
            m.word[at >> 5] |= 1u << (at & 31);
        }
    return m;
}

// ---- how the groups of a launch are shared out over its CTAs ------------------------------------------
// The packed groups of all sequences form one running list, and CTA i takes groups [i * per, (i + 1) * per) of it, whatever
// sequences they belong to (32 sequences of 1K..32K tokens in splits of 512 were 2048 CTAs in waves of 148, each with 7 to 9 us
// around its steady state: 560 us of store and decode against 318 us).  A piece of a sequence writes its partial result to
// workspace slot (its CTA - the first CTA of the sequence), and the caller's workspace has S slots per sequence, which bounds `per`
// from below: shares are even up to one group where S is generous, and longer, up to the longest sequence over S - 1, where it is not
// (8 sequences of 4K..32K tokens, both stages: 96 us with 64 slots, 133 us with the 18 of ommx_b200_auto_num_kv_splits).
// Equal splits per sequence, dealt out one by one (per = 0: item x is split x % S of sequence x / S), are taken instead
//   * where that bound makes the shares longer than S of them per sequence would be, and
//   * where a share could hold more sequences than a CTA lists (MAX_PIECES).  Of equal splits a CTA never has more than that:
//     stage1_grid makes a CTA for every MAX_PIECES of them as soon as there are that many sequences.  The line is drawn where any
//     lengths are safe; where none are short the list would have been, and is faster or slower (2 kv heads, S = 2: 187 sequences of
//     68..136 groups 115 us by the list, 173 by splits; 204 of 119..238 groups 341 and 226).  A line drawn from the shortest sequence
//     costs every batch: one more reduction ahead of the stages made the long cases 3 to 4 % slower.
// Where pieces begin depends on the plan, and with it the running maximum against which P is rounded to fp16: another split
// count or batch moves a result by about 5e-5 of its norm, the same call repeats its bits.
//
// Where S bounds the shares from below and leaves CTAs without one - few sequences in splits of
// 512 tokens - a share (or split) is worked on by a whole cluster of CTAs: each piece is dealt out evenly to them, and for every
// kv head one of them merges the others' softmax states through their shared memory before the one result goes to the piece's slot.
// It is taken where the groups per CTA, the merge counted as one more, get fewer.  Measured, 8 kv heads, without / with the size taken
// (2, 4, 8): 4K in 8 slots 42.2 / 18.5 us (28.6, 20.6, 18.1); 16K in 32 42.6 / 23.6 (28.9, 22.8, 24.8); 8 sequences of 700..2048 in 4
// 43.1 / 25.0 (31.1, 24.1, 33.1); 4 of 4K..8K in 16 43.0 / 32.3 (31.5, 33.3, 37.5).  In brackets before the barrier that holds
// a cluster's CTAs until all have read (0.4..0.9 us).
struct SharePlan {
    int per, total;                      // groups per share (0: equal splits per sequence), groups of all sequences
    int ctas, shares;                    // CTAs to a share, shares
};
__host__ __device__ __forceinline__ int groups_of(int seq) { return seq > 0 ? (seq + 31) >> 5 : 0; }
__host__ __device__ __forceinline__ SharePlan share_plan_of(int total, int longest, int B, int S, const Divisor &ncta, int waves, const ShareDivisors &by) {
    SharePlan s;
    s.total = total;
    s.ctas = 1;
    s.shares = (int)ncta.d;
    s.per = max(1, ncta.of(total + (int)ncta.d - 1));
    const int equal = by.slots.of(longest + S - 1);
    if (B == 1) {
        s.per = max(s.per, equal);                             // a lone sequence starts at a CTA's beginning: exactly ceil(n / per) slots
    } else {
        if (S >= 2) s.per = max(s.per, longest >= 2 ? by.slots1.of(longest - 2) + 1 : 1);   // anywhere else it touches up to (n - 2) / per + 2 CTAs
        if (S < 2 || min(s.per, B) > MAX_PIECES || (waves <= MAX_PIECES && waves * equal <= s.per)) s.per = 0;
    }
    return s;
}
__host__ __device__ __forceinline__ SharePlan share_plan_of(int total, int longest, int B, int S, const Stage1Grid &g, const ShareDivisors &by) {
    SharePlan a = share_plan_of(total, longest, B, S, by.ctas, g.waves, by);
    if (g.cluster > 1) {
        const int equal = by.slots.of(longest + S - 1);
        SharePlan c = share_plan_of(total, longest, B, S, by.shares, g.cluster_waves, by);
        c.ctas = g.cluster;
        const int of_a = a.per > 0 ? a.per : g.waves * equal, of_c = c.per > 0 ? c.per : g.cluster_waves * equal;
        if ((c.per > 0 || g.cluster_waves <= MAX_PIECES) && (of_c + g.cluster - 1) / g.cluster + 1 < of_a) return c;
    }
    return a;
}
// Host code without a device takes a chip of so many SMs to be a B200, which runs 74, 33 and 15 clusters on 148 (a launch asks its device)
static inline Chip chip_of(int sm_count) { return Chip{sm_count, {sm_count / 2, sm_count * 33 / 148, sm_count * 15 / 148}}; }
// CTAs of a launch - one per SM, or one per group where there are fewer; above MAX_PIECES sequences at least one for every MAX_PIECES
// groups or splits - and the rounds of them that equal splits would take (capped: past the cap they are never the choice)
static inline Stage1Grid stage1_grid(int batch, int S, int max_seq_len, const Chip &chip) {
    const int sm_count = chip.sms;
    const long long longest = groups_of(max_seq_len), groups = batch * longest, splits = (long long)batch * S;
    const long long least = batch > MAX_PIECES ? (max(groups, splits) + MAX_PIECES - 1) / MAX_PIECES : 1;
    Stage1Grid g;
    g.ncta = (int)max(min((long long)sm_count, max(groups, 1ll)), least);
    g.cluster = 1;
    // The cluster size that leaves the fewest groups per CTA if all sequences are of the longest's length; share_plan_of then decides by
    // the lengths.  No more clusters than run at once: on a B200's 148 SMs 74 of two, 33 of four, 15 of eight.  A launch that cannot
    // gain at equal lengths keeps the form without clusters: the exchange's code alone costs 4.5 % (8 x 32K: 133.9 -> 140.0 us), although
    // a ragged batch would win by more (8 sequences of 4K..32K in 18 slots each: 133.5 -> 103.4).
    if (batch <= MAX_PIECES && S > (batch > 1 ? 1 : 0)) {
        const long long bound = batch == 1 ? (longest + S - 1) / S : (longest - 2) / (S - 1) + 1;
        long long best = min(max((groups + sm_count - 1) / sm_count, bound), (splits + sm_count - 1) / sm_count * ((longest + S - 1) / S));
        for (int c = 2; c <= 8; c *= 2) {
            const long long at_once = chip.clusters[c / 4], shares = max(1ll, min(at_once, groups));
            if (at_once == 0) continue;
            const long long cost = (min(max((groups + shares - 1) / shares, bound), (splits + shares - 1) / shares * ((longest + S - 1) / S)) + c - 1) / c + 1;
            if (cost < best) { best = cost; g.cluster = c; g.ncta = (int)shares * c; }
        }
    }
    g.waves = (int)min((splits + g.ncta - 1) / g.ncta, 1024ll);
    const int shares = g.ncta / g.cluster;
    g.cluster_waves = (int)min((splits + shares - 1) / shares, 1024ll);
    return g;
}
// called by whole warps; every lane gets the same answer
template <bool CLUSTER>
__device__ __forceinline__ SharePlan share_plan(const int32_t *b_seq_len, int B, int S, const Stage1Grid &g, const ShareDivisors &by, int lane) {
    int n = 0, mx = 0;
    if (B == 1) {
        n = mx = groups_of(b_seq_len[0]);
    } else {
        for (int i = lane; i < B; i += 32) {
            const int g = groups_of(b_seq_len[i]);
            n += g;
            mx = max(mx, g);
        }
        n = __reduce_add_sync(0xFFFFFFFFu, n);
        mx = __reduce_max_sync(0xFFFFFFFFu, mx);
    }
    if constexpr (CLUSTER) return share_plan_of(n, mx, B, S, g, by);
    else return share_plan_of(n, mx, B, S, by.ctas, g.waves, by);
}

// One piece of work of a CTA: consecutive groups of one sequence.  `it` counts the CTA's ring stages across its pieces, so that
// the ring never drains between two of them.  One warp lists the pieces in shared memory; the roles walk that list, because
// the walk's own state costs a decode warp (56 registers) 9 % of its speed in spills.
struct alignas(16) Piece {
    int b, slot, g0, ng;                 // sequence, workspace slot, first group in the sequence, groups
    int ntok, it0, it1, more;            // tokens, ring iterations [it0, it1), whether another piece follows
};
struct PieceWalk {
    int pos, end, step;                  // running list: first group of the piece, end of this CTA's share; splits: item, items, items between two
};
template <int GS>
__device__ __forceinline__ void piece_range(Piece &c, int seq, int g0, int ng) {
    c.g0 = g0;
    c.ng = ng;
    c.ntok = min(seq - 32 * g0, 32 * ng);
    c.it1 = c.it0 + (ng + GS - 1) / GS;
}
// equal splits: the first item at or after w.pos that has groups
template <int GS> __device__ __forceinline__ bool piece_of_splits(Piece &c, PieceWalk &w, const S1Params &p) {
    for (; w.pos < w.end; w.pos += w.step) {
        c.b = w.pos / p.S;
        c.slot = w.pos - c.b * p.S;
        const int seq = p.b_seq_len[c.b], n = groups_of(seq), per = (n + p.S - 1) / p.S, g0 = c.slot * per;
        if (g0 < n) {
            piece_range<GS>(c, seq, g0, min(per, n - g0));
            return true;
        }
    }
    return false;
}
template <int GS> __device__ __forceinline__ bool first_piece(Piece &c, PieceWalk &w, const S1Params &p, const SharePlan &plan, int cta, int lane) {
    c.it0 = 0;                                                 // cta: the share
    if (plan.per == 0) {
        w.pos = cta;
        w.end = p.B * p.S;
        w.step = plan.shares;
        return piece_of_splits<GS>(c, w, p);
    }
    w.pos = cta * plan.per;
    w.end = min(w.pos + plan.per, plan.total);
    if (w.pos >= w.end) return false;
    int off = 0, seq, n;                                       // groups before the sequence that holds w.pos
    if (p.B == 1) {
        c.b = 0;
        seq = p.b_seq_len[0];
        n = groups_of(seq);
    } else {
        for (int base = 0;; base += 32) {
            const int len = base + lane < p.B ? p.b_seq_len[base + lane] : 0;
            const int g = groups_of(len);
            int x = g;                                         // inclusive sums over the lanes
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xFFFFFFFFu, x, o);
                if (lane >= o) x += y;
            }
            const uint32_t past = __ballot_sync(0xFFFFFFFFu, off + x > w.pos);
            if (past) {
                const int l = __ffs(past) - 1;
                c.b = base + l;
                seq = __shfl_sync(0xFFFFFFFFu, len, l);
                n = __shfl_sync(0xFFFFFFFFu, g, l);
                off += __shfl_sync(0xFFFFFFFFu, x, l) - n;
                break;
            }
            off += __shfl_sync(0xFFFFFFFFu, x, 31);
        }
    }
    c.slot = off > 0 ? cta - off / plan.per : cta;
    const int g0 = w.pos - off, ng = min(n - g0, w.end - w.pos);
    piece_range<GS>(c, seq, g0, ng);
    return true;
}
template <int GS> __device__ __forceinline__ bool next_piece(Piece &c, PieceWalk &w, const S1Params &p, const SharePlan &plan) {
    c.it0 = c.it1;
    if (plan.per == 0) {
        w.pos += w.step;
        return piece_of_splits<GS>(c, w, p);
    }
    w.pos += c.ng;
    if (w.pos >= w.end) return false;
    int seq;
    do seq = p.b_seq_len[++c.b];                               // the share has groups left, so a later sequence has some
    while (seq <= 0);
    const int n = groups_of(seq), ng = min(n, w.end - w.pos);
    c.slot = 0;                                                // it begins inside this CTA's share
    piece_range<GS>(c, seq, 0, ng);
    return true;
}

// The part of a piece that CTA `rank` of the `n` that share it works on, its ring iterations from `it0` on; there may be nothing in it.
// Which CTA gets the odd groups turns with the piece.
template <int GS> __device__ __forceinline__ Piece part_of(const Piece &c, int rank, int n, int it0) {
    Piece q = c;
    if (n > 1) {
        const int r = (rank + c.b + c.slot) % n, lo = c.ng * r / n;
        q.g0 = c.g0 + lo;
        q.ng = c.ng * (r + 1) / n - lo;
        q.ntok = min(c.ntok - 32 * lo, 32 * q.ng);
    }
    q.it0 = it0;
    q.it1 = it0 + (q.ng + GS - 1) / GS;
    return q;
}

constexpr size_t SMEM_LIMIT = 232448;   // what a CTA may ask for
constexpr size_t stage1_smem(int stages, int stage_bytes, int groups, int pages_per_group) {       // last line: copy roles, their table entries, pieces
    return 1024 + (size_t)stages * stage_bytes + (size_t)NCW * DT_BYTES + 64 + (2 * MAX_STAGES + (2 + MAX_STAGES) * NCW + 3 * NCW) * 8
           + (size_t)groups * (4 * pages_per_group + 6) * (sizeof(CopyDesc) + 4) + MAX_PIECES * sizeof(Piece);
}
// KOUT: outliers per K vector known at compile time (static, unrolled splice) or -1 (runtime).
//
// Every MMA is m16n8k16.  Logits in bf16: a 2-bit code field masked in place is a bf16 subnormal, code * 4^slot * 2^-133, exact and
// without an offset (subnormal operands run at full rate), and q, the factors 2^e and the deltas are bf16 as they are, so no
// product is rounded.  Output in fp16, whose subnormals hold a code field too (code * 4^slot * 2^-24) and whose 11 bits P needs.
// N = 8 columns are the query heads of the kv head (GQA <= 8).
//   logits   S^T[token][head]  = codes[token][ch] . (q * 2^e_k)[ch][head]      (2 m-tiles x 8 k-steps)
//                              + delta[token][ch] . q[ch][head]                (sidecar tile, same shape)
//                              + zp[ch] . q[ch][head]                          (one row, broadcast)
//   output   O^T[ch][head]     = codes^T[ch][token] . (P * 2^e_v)[token][head] (8 m-tiles x 2 k-steps, the
//                                16 rows of an m-tile lie in one V scale group)
//                              + vz^T[group][token] . P[token][head]
// The power-of-two factors and deltas of a unit are laid out for these fragments by the decode warps (the sidecar tile), so the MMA
// warps multiply and accumulate and do little else; q.zp, which they compute themselves, fits into their wait for the deltas, and the
// V zero-points come straight out of the staged plane by a transposed ldmatrix.
//
// Bound by issue slots, the logic pipe and shared-memory wavefronts (399 of them and 1536 instructions per unit, near four fifths of
// what pipe and slots can do in the steady state), which both roles share: leaving out any part of either saves its share, and the MMA warps' chain of code
// MMAs, delta MMAs, softmax and P.V stands close behind.  The register file (8 x 128 + 16 x 56 a lane) holds no second unit in
// flight, and memory is at 28 to 32 % of its rate.  Logits in bf16 (the deltas need no second conversion), one packed min-max-add per
// factor pair, V factors by one warp with lane = token and zero-points without staging, code words by ldmatrix, zero-point words
// used as loaded, and a maximum that follows lazily, before -> with them, this stage and stage 2: 64K x 8 heads 44.8 -> 41.8 us;
// 8 x 32K, 70B heads 148.7 -> 136.4; 32 sequences of 1K to 32K in splits of 512 with the store 318 -> 291.5.
// Tried and slower (64K / 70B): 16 warps that each build and use their own half tile, no hand-overs (47.2 / 162 us, latency-bound
// at four warps a scheduler); 16 delta warps with their own MMAs beside 8 output warps (46.1 / 167); tile rows zeroed by an
// out-of-range tensor-map load (83 / 289); FP4 levels by the conversion instruction and a shorter wait loop (53 fewer
// instructions per unit, same time).
// With one or two kv heads a unit costs more: 1856 and 1692 instructions and 428 and 448 wavefronts (103 and 139 of them bank conflicts,
// 111 at eight heads), because a token row of theirs is 32 or 64 bytes, staged without a swizzle, and a stage has eight or four groups.
// PLAIN: the recipes that are served - bitmask or relidx7 index, outlier map, no logit cap, no differential-timing knob, a page layout that
// leaves room for the usual ring depth - with every choice between those made at compile time, plane offsets included.  The general
// form keeps them at run time; its tests and address arithmetic inside the unit cost it 12 to 15 % (both stages: 64K
// 46.1 us against 41.0, 70B heads 8 x 32K 155.4 against 135.5).
// IDX7 (plain form only): relidx7 positions instead of bitmasks, turned into masks by three instructions a position.  At run time, byte
// by byte, they took longer than the rest of the tile: 64K x 8 heads, both stages, k = 6 66.3 -> 45.9 us, k = 12 94.9 -> 58.7.
template <int KOUT, int H, bool IDX7> struct PlainLayout {
    static constexpr bool GATHER = H <= 4;
    static constexpr int GS = NCW / H;
    static constexpr int U = GATHER ? NCW : H;                       // units to a block
    static constexpr int NB = KOUT > 0 ? (KOUT + 1) / 2 : 0, NBI = IDX7 ? (7 * KOUT + 7) / 8 : 4;
    static constexpr int VM = U * 1024, VS = U * 2048, VZ = VS + U * 128, KS = VZ + U * 256, KZ = KS + U * 128, MS = KZ + U * 256, MC = MS + U * 256,
                         BM = MC + U * 256, OV = BM + U * 128 * NBI;
    static constexpr int GB = (OV + U * 128 * NB + 1023) / 1024 * 1024;
    static constexpr int STAGE = NCW / U * GB;
    static constexpr int STAGES = stage1_smem(4, STAGE, GS, 2) <= SMEM_LIMIT ? 4 : 3;   // with 16-token pages
    static_assert(stage1_smem(STAGES, STAGE, GS, 2) <= SMEM_LIMIT, "the ring fits");
    // Copies of four rows.  A row is a group slot, half of one at four heads; for page planes a page, or half of one where a stage has
    // two.  The code planes of four heads go by page, swizzled, as does slot by slot an outlier index whose rows would be too long.
    static constexpr int CODE_ROWS = H == 4 ? 1 : 4, SLOT_SPLIT = gather_slot_split(H), SLOT_ROWS = GS * SLOT_SPLIT;
    static constexpr bool ROWS_FIT = H * 128 * NBI / SLOT_SPLIT <= GATHER_ROW_MAX;
    static constexpr int GROUP_COPIES = (KOUT == 0 ? 2 : 6) * (SLOT_ROWS / 4) + (ROWS_FIT ? 0 : GS - SLOT_ROWS / 4);
    static __host__ __device__ constexpr int copies(int pages) {
        return 2 * (pages / CODE_ROWS) + 2 * (pages * gather_page_split(pages) / 4) + GROUP_COPIES;
    }
};
template <int H, bool PLAIN> struct Stage1Form {
    static constexpr bool GATHER = PLAIN && H <= 4;
    typedef WarpLayout<H, GATHER> Layout;
    typedef std::conditional_t<GATHER, S1GatherParams, S1Params> Params;
};
template <int KOUT, int H, bool PLAIN, bool IDX7, bool CLUSTER>
__global__ void __launch_bounds__(Stage1Form<H, PLAIN>::Layout::THREADS, 1)
decode_stage1_kernel(const __grid_constant__ typename Stage1Form<H, PLAIN>::Params p) {
    constexpr bool GATHER = Stage1Form<H, PLAIN>::GATHER;
    typedef typename Stage1Form<H, PLAIN>::Layout Warps;
    constexpr bool WIDE = Warps::WIDE;
    constexpr int NDW = Warps::NDW, NPW = Warps::NPW, PRODUCER_WARP = Warps::PRODUCER_WARP;
    constexpr int S1_THREADS = Warps::THREADS;
    constexpr int GS = NCW / H;                                     // groups per ring stage
    constexpr int TS = H * 32;                                      // bytes per token row (all heads)
    constexpr uint32_t SWZ = H >= 4 ? 0x70u : 0u;    // the code planes are staged through swizzled tensor maps
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // swizzle atoms are 1 KB: align the ring by hand (the launch adds 1 KB of slack)
    uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int cta = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    static_assert(!PLAIN || KOUT >= 0, "the plain form knows its outlier count");
    typedef PlainLayout<KOUT, H, IDX7> L;
    const int NS = PLAIN ? L::STAGES : p.nstages;
    const int gb_bytes = PLAIN ? L::GB : p.gb_bytes, stage_bytes = PLAIN ? L::STAGE : p.stage_bytes;
    const int o_vm = PLAIN ? L::VM : p.o_vm, o_vs = PLAIN ? L::VS : p.o_vs, o_vz = PLAIN ? L::VZ : p.o_vz, o_ks = PLAIN ? L::KS : p.o_ks,
              o_kz = PLAIN ? L::KZ : p.o_kz, o_ms = PLAIN ? L::MS : p.o_ms, o_mc = PLAIN ? L::MC : p.o_mc, o_bm = PLAIN ? L::BM : p.o_bm,
              o_ov = PLAIN ? L::OV : p.o_ov;
    const int abl = PLAIN ? 0 : p.abl;
    const bool use_map = PLAIN || p.use_map, idx7 = PLAIN ? IDX7 : p.idx7;
    const int k_out = KOUT >= 0 ? KOUT : p.k_out;
    const long long wait_limit = (abl & ABL_TEST_STALL) ? TEST_WAIT_LIMIT_CYCLES : WAIT_LIMIT_CYCLES;

    // ---- shared memory carve-up ----
    uint8_t *s_stage = smem;                                            // nstages * stage_bytes
    uint8_t *s_tiles = s_stage + NS * stage_bytes;                    // NCW * DT_BYTES
    float *s_lut = reinterpret_cast<float *>(s_tiles + NCW * DT_BYTES);
    uint64_t *s_bar = reinterpret_cast<uint64_t *>(s_lut + 16);         // full[], empty[], tile_full[NCW], tile_empty[NCW][], tile_rows[NCW]
    CopyDesc *s_desc = reinterpret_cast<CopyDesc *>(s_bar + 2 * MAX_STAGES + (5 + MAX_STAGES) * NCW);
    const uint32_t bar_full = smem_u32(s_bar), bar_empty = smem_u32(s_bar + MAX_STAGES);
    const uint32_t bar_tfull = smem_u32(s_bar + 2 * MAX_STAGES), bar_tempty = smem_u32(s_bar + 2 * MAX_STAGES + NCW);
    const uint32_t bar_trows = smem_u32(s_bar + 2 * MAX_STAGES + (1 + MAX_STAGES) * NCW);
    // states of a head: handed in by the cluster's other CTAs, taken from this one; whether there is one (8 bytes a head)
    const uint32_t bar_handed = bar_trows + 8 * NCW, bar_taken = bar_handed + 8 * NCW, s_there = bar_taken + 8 * NCW;
    volatile int *s_ctas = reinterpret_cast<int *>(s_bar + 2 * MAX_STAGES + (4 + MAX_STAGES) * NCW) + 1;   // CTAs to a share (the odd word of s_there[0])

    // ---- prologue: LUT, barriers and copy descriptors.  None of it depends on an earlier kernel, so it runs while the
    //      kernel before this one in the stream drains (the grid may start then, see the wait below). ----
    // the first tensor-map copy otherwise pays for fetching its descriptor
    if (SWZ != 0 && threadIdx.x == S1_THREADS - 32) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&p.tmap_k)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&p.tmap_v)) : "memory");
    }
    if constexpr (GATHER) {
        const int i = (int)threadIdx.x - (S1_THREADS - 32);
        if (i >= (L::CODE_ROWS == 1 ? 2 : 0) && i < (KOUT > 0 ? 10 : 6) && (i != 8 || L::ROWS_FIT))
            asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&p.rows[i])) : "memory");
    }
    // the sidecar tiles: rows that no half writes stay zero
    for (int i = threadIdx.x; i < NCW * DT_BYTES / 16; i += S1_THREADS) reinterpret_cast<uint4 *>(s_tiles)[i] = make_uint4(0, 0, 0, 0);
    if (threadIdx.x < 16) {
        const int c = threadIdx.x;
        const int mi = ((c >> 1) & 3) * 2 + (c & 1);                    // exp*2 + mant
        const float mag = mi == 0 ? 0.f : (mi == 1 ? .5f : (float)(2 + (mi & 1)) * (float)(1 << (mi >> 1)) * 0.25f);
        s_lut[c] = (c & 8) ? -mag : mag;
    }
    {
        // one barrier per thread (72 of them: a single thread's serial inits were a microsecond of every launch)
        const int t = (int)threadIdx.x - 32;
        constexpr int NB_RING = 2 * MAX_STAGES, NB_TILE = NB_RING + (2 + MAX_STAGES) * NCW, NB_ALL = NB_TILE + (CLUSTER ? 2 * NCW : 0);
        if (t >= 0 && t < NB_ALL) {
            uint32_t count;
            if (t < MAX_STAGES) count = NPW;                                   // full[]: each producer warp announces its own copies
            else if (t < NB_RING) count = 3 * NCW;                             // empty[]: 8 MMA warps + 16 tile halves
            else if (t < NB_RING + NCW) count = 2;                             // tile_full[]: the two halves' deltas scattered
            else if (t < NB_RING + NCW + MAX_STAGES * NCW) count = 1;          // tile_empty[][]
            else if (t < NB_TILE) count = 2;                                   // tile_rows[]: the two halves' rows written
            else if (t < NB_TILE + NCW) count = max(p.grid.cluster - 1, 1);    // handed[]: by every other CTA of the cluster
            else count = 1;                                                    // taken[]
            mbar_init(bar_full + 8 * t, count);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    }
    const int cpg = 4 * p.ppg + 6;                                      // copies per group
    const int ppg_log = __ffs(p.ppg) - 1, stage_pages = GS << ppg_log;
    const int page_split = H == 4 ? gather_page_split(stage_pages) : 1, page_rows = stage_pages * page_split;
    const int ncopies = GATHER ? L::copies(stage_pages) : GS * cpg;
    if constexpr (GATHER) {
        const int c = (int)threadIdx.x - 64;
        const int n_code = 2 * (stage_pages / L::CODE_ROWS), n_page = n_code + 2 * (page_rows / 4);
        if (c >= 0 && c < ncopies) {
            int plane, row;                                             // its first row
            if (c < n_code) {
                plane = c >= n_code / 2;
                row = L::CODE_ROWS * (c - plane * (n_code / 2));
            } else if (c < n_page) {
                plane = 2 + (c >= (n_code + n_page) / 2);
                row = 4 * (c - (plane == 2 ? n_code : (n_code + n_page) / 2));
            } else {
                const int x = c - n_page;
                constexpr int Q = L::SLOT_ROWS / 4, FIRST = 4 * Q;      // k_scale, k_zp, map scale, map center; then index, values
                constexpr int Q8 = L::ROWS_FIT ? Q : GS;
                plane = x < FIRST ? 4 + x / Q : (x < FIRST + Q8 ? 8 : 9);
                row = plane < 8 ? 4 * (x % Q) : (plane == 8 ? (L::SLOT_ROWS / Q8) * (x - FIRST) : 4 * (x - FIRST - Q8));
            }
            const bool by_page = plane < 4, single = (plane < 2 && L::CODE_ROWS == 1) || (plane == 8 && !L::ROWS_FIT);
            const int split = by_page ? (plane < 2 ? 1 : page_split) : L::SLOT_SPLIT;
            const uint32_t bytes = (by_page ? (uint32_t)p.ps * H * (plane < 2 ? 32u : (plane == 2 ? 4u : 8u))     // of a row
                                            : H * 128u * (plane == 4 ? 1u : (plane < 8 ? 2u : (plane == 8 ? (uint32_t)L::NBI : (uint32_t)L::NB)))) >> (split - 1);
            const uint32_t at[10] = {0, L::VM, L::VS, L::VZ, L::KS, L::KZ, L::MS, L::MC, L::BM, L::OV};
            uint32_t off = 0;
#pragma unroll
            for (int i = 1; i < 10; ++i) off = plane == i ? at[i] : off;
            CopyDesc d;
            d.src = p.k_obmp;                                           // of the one plane that may be copied slot by slot
            d.unit = bytes * (single ? (plane == 8 ? L::SLOT_SPLIT : 1) : 4);
            d.dst = off + row * bytes;
            d.tbase = plane < 2 ? row * page_split : (by_page ? row : page_rows + row);
            d.tmul = 0;
            const int whole = row >> (split - 1), gi = by_page ? whole >> ppg_log : whole;   // page or slot, its group
            d.tok0 = by_page ? (whole & (p.ppg - 1)) * p.ps : 0;
            d.gi = gi | (single ? (plane < 2 ? plane + 1 : 0) : 3 + plane) << 8;
            s_desc[c] = d;
        }
    } else {
        // Copy roles (group-in-stage, plane) are tabulated once; the producer's loop body is then one
        // descriptor load, one multiply-add and one copy per role, with no divergent paths, because that
        // single warp's issue latency bounds how fast stages refill.
        const uint32_t page_b = (uint32_t)p.ps * H;                     // (token, head) rows per page
        const int c = (int)threadIdx.x - 64;                            // threads 64.. build one descriptor each
        if (c >= 0 && c < ncopies) {
            CopyDesc d;
            d.src = nullptr; d.unit = 0; d.dst = 0; d.tbase = 0; d.tmul = 0; d.gi = 0; d.tok0 = 0;
            const int gi = c / cpg, ci = c - gi * cpg;
            d.gi = gi;
            const uint32_t gbo = (uint32_t)gi * gb_bytes;
            if (ci < 4 * p.ppg) {
                const int pg = ci >> 2, plane = ci & 3;
                const uint32_t w = plane < 2 ? 32u : (plane == 2 ? 4u : 8u);
                d.src = plane == 0 ? p.k_base : (plane == 1 ? p.v_main : (plane == 2 ? p.v_scale : p.v_zp));
                d.unit = page_b * w;
                d.dst = gbo + (plane == 0 ? 0u : (plane == 1 ? (uint32_t)o_vm : (plane == 2 ? (uint32_t)o_vs : (uint32_t)o_vz)))
                      + (uint32_t)pg * page_b * w;
                d.tbase = pg; d.tmul = p.ppg; d.tok0 = pg * p.ps;
                if (SWZ != 0 && plane < 2) d.gi |= (plane + 1) << 8;
            } else {
                const int gp = ci - 4 * p.ppg;
                const bool on = gp < 2 || (k_out > 0 && (gp >= 4 || use_map));
                if (on) {
                    const uint32_t w = gp == 0 ? 128u : (gp == 4 ? 128u * p.nbi : (gp == 5 ? 128u * p.nb : 256u));
                    d.src = gp == 0 ? p.k_scale : (gp == 1 ? p.k_zp : (gp == 2 ? p.k_ms : (gp == 3 ? p.k_mc : (gp == 4 ? p.k_obmp : p.k_oval))));
                    d.unit = (uint32_t)H * w;
                    d.dst = gbo + (uint32_t)(gp == 0 ? o_ks : (gp == 1 ? o_kz : (gp == 2 ? o_ms : (gp == 3 ? o_mc : (gp == 4 ? o_bm : o_ov)))));
                    d.tbase = 0; d.tmul = 0;                            // tmul 0: the index is a group slot
                }
            }
            s_desc[c] = d;
        }
    }
    __syncthreads();
    if constexpr (CLUSTER) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");         // this CTA's barriers are ready
    Piece pc;
    Piece *s_piece = reinterpret_cast<Piece *>(s_desc + GS * cpg);
    auto wait_for_earlier_kernels = [&]() __attribute__((always_inline)) {
        // Nothing an earlier kernel may have written - lengths, tables, the query, the planes, the split workspace a
        // previous layer's combine still reads - is touched before this returns.
        asm volatile("griddepcontrol.wait;" ::: "memory");
        // Stage 2 is launched as a programmatic dependent: it may start its own prologue (residual-row
        // logits, which do not depend on this kernel but may depend on the one before it: hence after the wait)
        // as soon as SM resources free up, and waits for this grid to finish before it reads the split partials.
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    };
    // The list of pieces is there (and the first ring fill on its way); false: this CTA has none.
    int pi = 0;
    auto pieces_listed = [&]() __attribute__((always_inline)) {
        asm volatile("bar.sync 0, %0;" ::"n"(S1_THREADS) : "memory");
        if constexpr (CLUSTER) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        pc = s_piece[0];
        return pc.b >= 0;
    };
    auto step_piece = [&]() __attribute__((always_inline)) {
        if (!pc.more) return false;
        pc = s_piece[++pi];
        return true;
    };

    const int g = lane >> 2, j = lane & 3;
    const float LOG2E = 1.4426950408889634f;
    const bool no_outlier = (abl & ABL_NO_OUTLIER) != 0;

    // ---- one stage of the ring: look up its page ids and group slots, announce its bytes, issue its copies (producer
    //      warps).  The lookup of a stage runs while the stage before it is still on its way, so that no copy waits for its
    //      table entry; each lane leaves what it finds in s_idx for itself. ----
    // (four rows to a copy make fewer descriptors, and four warps' entries fit behind them)
    int32_t *s_idx = GATHER ? reinterpret_cast<int32_t *>(s_desc + ncopies) : reinterpret_cast<int32_t *>(s_piece + MAX_PIECES);
    auto whole_stage = [&](const Piece &q, int it) { return 32 * GS * (it + 1 - q.it0) <= q.ntok; };
    auto copy_on = [&](const CopyDesc &d, const Piece &q, int it) __attribute__((always_inline)) {
        const int lg = (it - q.it0) * GS + (d.gi & 0xFF);
        return d.unit != 0 && lg < q.ng && 32 * lg + d.tok0 < q.ntok;
    };
    auto lookup_stage = [&](const Piece &q, int it, int nshare, int share) __attribute__((always_inline)) {
        const int64_t g0 = (int64_t)p.seg_group_base + q.g0 + (it - q.it0) * GS;
        if constexpr (GATHER) {
            // every page and slot of the stage once (or twice, its halves); what the sequence does not have there repeats the first,
            // so that a copy of four rows reads nothing else
            int32_t *idx = s_idx + share * (page_rows + L::SLOT_ROWS);
            __syncwarp();                                           // the last stage's have been read
            for (int i = lane; i < page_rows + L::SLOT_ROWS; i += 32) {
                const bool page = i < page_rows;
                const int split = page ? page_split : L::SLOT_SPLIT, x = (page ? i : i - page_rows) >> (split - 1);   // page or slot of the stage
                const int gi = page ? x >> ppg_log : x, pg = page ? x & (p.ppg - 1) : 0, lg = (it - q.it0) * GS + gi;
                const bool on = lg < q.ng && 32 * lg + pg * p.ps < q.ntok;
                const int64_t at = page ? (int64_t)q.b * p.r2t_sb + g0 * p.ppg + (on ? x : 0) : (int64_t)q.b * p.r2g_sb + g0 + (on ? x : 0);
                int64_t id = load_index(page ? p.r2t : p.r2g, p.tbl64, at);
                if (id < 0 || id >= (page ? p.num_pages : p.num_slots)) { or_status(p.status, page ? OMMX_ST_BAD_PAGE : OMMX_ST_BAD_GROUP); id = 0; }
                idx[i] = (int)id * split + ((page ? i : i - page_rows) & (split - 1));
            }
            __syncwarp();
            return;
        }
#pragma unroll 1
        for (int ci = lane * nshare + share; ci < ncopies; ci += 32 * nshare) {
            const CopyDesc d = s_desc[ci];
            if (!copy_on(d, q, it)) continue;
            const bool page = d.tmul != 0;                          // tmul 0: the index is a group slot
            const int64_t at = page ? (int64_t)q.b * p.r2t_sb + (g0 + (d.gi & 0xFF)) * d.tmul + d.tbase : (int64_t)q.b * p.r2g_sb + g0 + (d.gi & 0xFF);
            int64_t x = load_index(page ? p.r2t : p.r2g, p.tbl64, at);
            if (x < 0 || x >= (page ? p.num_pages : p.num_slots)) { or_status(p.status, page ? OMMX_ST_BAD_PAGE : OMMX_ST_BAD_GROUP); x = 0; }
            s_idx[ci] = (int)x;
        }
    };
    // `nshare` warps split the copies of a stage, this one taking share `share`; with `announce_all` it announces the bytes
    // of all of them (the others then announce nothing), else its own.
    // (A copy of another warp may land before the announcement: the phase cannot complete without the announcing arrival,
    // and the transaction count may run negative meanwhile.)
    auto stage_bytes_of = [&](const Piece &q, int it, bool whole, int first, int step) __attribute__((always_inline)) {
        uint32_t mine = 0;
#pragma unroll 1
        for (int ci = first; ci < ncopies; ci += step) {
            const CopyDesc d = s_desc[ci];
            if (whole || copy_on(d, q, it)) mine += d.unit;
        }
        return __reduce_add_sync(0xFFFFFFFFu, mine);
    };
    auto issue_stage = [&](const Piece &q, int it, int nshare, int share, bool announce, uint32_t bytes) __attribute__((always_inline)) {
        const int s = ring_slot(it, NS);
        if (announce) {
            if (lane == 0) mbar_arrive_expect_tx(bar_full + 8 * s, bytes);
            __syncwarp();
        }
        const uint32_t sbase = smem_u32(s_stage + (size_t)s * stage_bytes);
#pragma unroll 1
        for (int ci = lane * nshare + share; ci < ncopies; ci += 32 * nshare) {
            const CopyDesc d = s_desc[ci];
            const int kind = d.gi >> 8;
            if (copy_on(d, q, it) && !((abl & ABL_TEST_STALL) && it == 1)) {
                if constexpr (GATHER) {
                    const int32_t *at = s_idx + share * (page_rows + L::SLOT_ROWS) + d.tbase;
                    if (L::CODE_ROWS == 1 && (kind == 1 || kind == 2)) {
                        tma_2d_g2s(sbase + d.dst, kind == 1 ? &p.tmap_k : &p.tmap_v, 0, *at * (p.rows_per_page >> (page_split - 1)), bar_full + 8 * s);
                    } else if (!L::ROWS_FIT && kind == 0) {
                        bulk_g2s(sbase + d.dst, d.src + (int64_t)*at * (d.unit / L::SLOT_SPLIT), d.unit, bar_full + 8 * s);
                    } else {
                        tma_rows_g2s(sbase + d.dst, &p.rows[kind - 3], *reinterpret_cast<const int4 *>(at), bar_full + 8 * s);
                    }
                    continue;
                }
                const int idx = s_idx[ci];
                if (kind == 0) bulk_g2s(sbase + d.dst, d.src + (int64_t)idx * d.unit, d.unit, bar_full + 8 * s);
                else tma_2d_g2s(sbase + d.dst, kind == 1 ? &p.tmap_k : &p.tmap_v, 0, idx * p.rows_per_page, bar_full + 8 * s);
            }
        }
    };
    // ---- what the producers do before the other roles start: deal out the work, fill the ring's first stage, list the pieces ----
    // The first fill is on every CTA's critical path.  A warp issues a bulk copy only about every 60 cycles and different warps
    // overlap, so in the narrow layout the three decode warps of the producer's warpgroup (idle until the data lands) take a
    // quarter of the first fill each.
    constexpr int FILL_WARP = PRODUCER_WARP - (WIDE ? 0 : 3);
    auto start_pieces = [&](const ShareDivisors &by) __attribute__((always_inline)) {
        PieceWalk walk;
        const SharePlan plan = share_plan<CLUSTER>(p.b_seq_len, p.B, p.S, p.grid, by, lane);
        auto my_part = [&](const Piece &c, int it0) __attribute__((always_inline)) {
            if constexpr (CLUSTER) return part_of<GS>(c, cluster_rank(), plan.ctas, it0);
            else return c;
        };
        if (!first_piece<GS>(pc, walk, p, plan, CLUSTER ? cta / plan.ctas : cta, lane)) {
            if (warp == PRODUCER_WARP && lane == 0) s_piece[0].b = -1;
            return;
        }
        Piece q = my_part(pc, 0);
        if (CLUSTER && q.ng == 0) {                                             // this CTA begins with a later piece, if any
            Piece c = pc;
            PieceWalk w = walk;
            while (q.ng == 0 && next_piece<GS>(c, w, p, plan)) q = my_part(c, 0);
        }
        if (!CLUSTER || q.ng > 0) {
            lookup_stage(q, 0, 4, warp - FILL_WARP);
            const uint32_t bytes = WIDE ? stage_bytes_of(q, 0, false, lane * NPW + warp - FILL_WARP, 32 * NPW)
                                        : (warp == PRODUCER_WARP ? stage_bytes_of(q, 0, false, lane, 32) : 0u);
            issue_stage(q, 0, 4, warp - FILL_WARP, WIDE || warp == PRODUCER_WARP, bytes);
        }
        if (warp == PRODUCER_WARP) {
            if (CLUSTER && lane == 0) *s_ctas = plan.ctas;
            int n = 0, at = 0;
            for (bool more = true; more; ++n) {
                Piece cur = my_part(pc, at);
                at = cur.it1;
                more = next_piece<GS>(pc, walk, p, plan);
                if (more && n + 1 == MAX_PIECES) {                       // a bounds check: share_plan_of rules it out
                    if (lane == 0) or_status(p.status, OMMX_ST_BAD_LENGTH);
                    more = false;
                }
                cur.more = more;
                if (lane == 0) s_piece[n] = cur;
            }
        }
    };

    // ---- one work item of the decode role: half hf of the sidecar tile of (iteration it, unit) ----
    // Channel 64 w + 16 j + 8 x + i (i = 0..7) sits in member x of the pair in register 8 w + i of lane group j in the MMAs
    // below, i.e. in column byte 128 w + 16 i + 4 j + 2 x of the delta rows.  This half has w = hf, this lane channels
    // 2 cp and 2 cp + 1 of it (the pair that code_bit_planes gives it): j = dj, x = dh, i = 2 da and 2 da + 1.
    const int cp = 8 * (lane & 2) + 2 * (lane >> 2) + (lane & 1);
    const int da = cp & 3, dh = (cp >> 2) & 1, dj = cp >> 3;
    const int lm_tok = 8 * ((lane >> 2) & 3) + 4 * (lane >> 4) + (lane & 3);
    // Build the sidecar tile of a unit between two uses by its MMA warp.  A tile is built in two
    // halves by two warps at once, because the MMA warp of the unit waits for it: half hf takes 64 of the
    // K channels (delta columns, scale factors), half 0 the V factors of all 32 tokens as well (lane = token).
    // Returns false when a bounded wait ran out.
    uint32_t e_max = 0;                                          // largest scale exponents seen, biased by 128, two halves
    auto decode_item = [&](const Piece &pc, const int n) __attribute__((always_inline)) -> bool {
        const int it = n / (2 * NCW), unit = (n >> 1) % NCW, hf = n & 1;
        const int h = unit % H, gsel = unit / H;
        uint8_t *tile = s_tiles + unit * DT_BYTES;
        const int s = ring_slot(it, NS);
        const uint32_t ph = ring_phase(it, NS);
        if (!mbar_wait(bar_full + 8 * s, ph, wait_limit)) {
            if (lane == 0) or_status(p.status, OMMX_ST_TIMEOUT);
            return false;
        }
        const int lg = (it - pc.it0) * GS + gsel;                 // local group of this unit
        const bool active = lg < pc.ng && !(abl & ABL_NO_COMPUTE);
        // (plane-major stages: group planes of units one after the other, token rows of group after group)
        const uint8_t *gb = s_stage + (size_t)s * stage_bytes + (GATHER ? 0 : (size_t)gsel * gb_bytes);
        const int hu = GATHER ? unit : h;
        const int d0 = 64 * hf + 2 * cp;                         // first of this lane's two channels
        const bool splice = k_out > 0 && !no_outlier;
        // ---- everything that only reads the stage comes before the wait for the tile, which the MMA warps make a decode warp
        //      wait for (a sixth of its time): the parameters of both channels, the K and V factors ----
        uint32_t e2 = 0, z2 = 0, kf = 0, f02 = 0, f13 = 0, ms2 = 0, mc2 = 0;
        uint2 bm2 = make_uint2(0u, 0u);
        // From 6 outliers on the base codes are looked up in bit planes in registers: a gather per outlier costs 3 to 4 conflicting
        // shared-memory wavefronts, the planes of 64 channels about 50 instructions.  64K x 8 heads, stage 1: k = 12 53.8 -> 50.2 us,
        // k = 8 43.3 -> 42.7, k = 6 40.3 -> 40.0; k = 4 37.2 -> 37.4 and k = 2 34.7 -> 35.5, which therefore gather.
        constexpr bool PLANES = KOUT >= 6 && KOUT % 2 == 0;
        uint32_t cw[4] = {0, 0, 0, 0};                           // bit planes of both channels' codes
        // Row pz of the code bytes of the channels at byte o of the head: byte pz*TS + h*32 + o of the (1 KB aligned) k_base
        // block, with the 16-byte chunk bits XOR-ed by the row's swizzle term.  h*32 + o splits into a part above
        // bit 7 (added to the row) and a part below (the XOR operand, swizzle term of the former included).
        const uint8_t *k_hi = gb + (GATHER ? gsel * H * 1024 : (h >> 2) * 128);
        const uint32_t k_sw = ((uint32_t)(h >> 2) * 16u) & SWZ;
        uint32_t st[2] = {0, 0}, sth[2] = {0, 0};                // nibble stream of each channel: outliers 0..7, 8..15
        if (active) {
            e2 = *reinterpret_cast<const uint16_t *>(gb + o_ks + hu * 128 + d0);
            z2 = *reinterpret_cast<const uint32_t *>(gb + o_kz + hu * 256 + 2 * d0);
            {
                // K scale factors 2^(e + KF_BIAS) * 4^-slot of the two channels, bf16
                const uint32_t eb = __byte_perm(e2 ^ 0x8080u, 0u, 0x4140u);                       // e + 128, two halves
                e_max = __vmaxs2(e_max, eb);
                const uint32_t off = da & 1 ? half2_const(KF_BIAS - 5, KF_BIAS - 7) : half2_const(KF_BIAS - 1, KF_BIAS - 3);
                const uint32_t top = da & 1 ? half2_const(E_TOP + KF_BIAS - 5, E_TOP + KF_BIAS - 7) : half2_const(E_TOP + KF_BIAS - 1, E_TOP + KF_BIAS - 3);
                kf = __viaddmin_s16x2(eb, off, top) << 7;
            }
            if (hf == 0) {
                // V scale factors 2^(e + FBIAS), fp16, of the four scale groups; lane = token
                const uint32_t w = 32 * lg + lane < pc.ntok ? *reinterpret_cast<const uint32_t *>(gb + o_vs + (GATHER ? gsel * H * 128 : 0) + (lane * H + h) * 4) ^ 0x80808080u : 0u;
                const uint32_t e02 = w & 0x00FF00FFu, e13 = (w >> 8) & 0x00FF00FFu;               // e + 128, groups 0, 2 and 1, 3
                e_max = __vimax3_s16x2(e_max, e02, e13);
                f02 = __viaddmin_s16x2_relu(e02, half2_const(FBIAS + 15 - 128, FBIAS + 15 - 128), half2_const(30, 30)) << 10;
                f13 = __viaddmin_s16x2_relu(e13, half2_const(FBIAS + 15 - 128, FBIAS + 15 - 128), half2_const(30, 30)) << 10;
            }
            if (splice) {
                if (use_map) {
                    ms2 = *reinterpret_cast<const uint32_t *>(gb + o_ms + hu * 256 + 2 * d0);
                    mc2 = *reinterpret_cast<const uint32_t *>(gb + o_mc + hu * 256 + 2 * d0);
                }
                if (!idx7) {
                    bm2 = *reinterpret_cast<const uint2 *>(gb + o_bm + hu * 512 + 4 * d0);
                } else {
                    // relidx7 (attention/codec.py:91-130 of the reference): k ascending token positions, 7 bits each,
                    // LSB first; the outlier set as a bitmask again, the value stream is shared with that encoding
                    uint32_t m2[2] = {0u, 0u};
                    if constexpr (KOUT > 0) {
                        // both channels' streams are 2 * NBI bytes back to back, 4-byte aligned where that is whole words
                        constexpr int NBI = (7 * KOUT + 7) / 8, NW = (2 * NBI + 3) / 4;
                        constexpr PositionBits PAST = past_31_bits(KOUT, NBI);
                        const uint8_t *ip = gb + o_bm + (hu * 128 + d0) * NBI;
                        uint32_t w[NW + 1] = {}, past = 0u;
                        if constexpr (NBI % 2 == 0) {
#pragma unroll
                            for (int i = 0; i < NW; ++i) w[i] = reinterpret_cast<const uint32_t *>(ip)[i];
                        } else {
#pragma unroll
                            for (int i = 0; i < NBI; ++i) w[i >> 1] |= (uint32_t)reinterpret_cast<const uint16_t *>(ip)[i] << (16 * (i & 1));
                        }
#pragma unroll
                        for (int i = 0; i < NW; ++i) past |= w[i] & PAST.word[i];
#pragma unroll
                        for (int c = 0; c < 2; ++c)
#pragma unroll
                            for (int r = 0; r < KOUT; ++r) {
                                const int bp = 8 * NBI * c + 7 * r;
                                m2[c] |= __funnelshift_l(0u, 1u, __funnelshift_r(w[bp >> 5], w[(bp >> 5) + 1], bp & 31));   // 1 << its low five bits
                            }
                        if (past) m2[0] = m2[1] = 0u;                    // reported below: no mask of k bits
                    } else {
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            const uint8_t *ip = gb + o_bm + (hu * 128 + d0 + c) * p.nbi;
                            uint32_t w[5] = {0u, 0u, 0u, 0u, 0u};
                            for (int i = 0; i < p.nbi; ++i) w[i >> 2] |= (uint32_t)ip[i] << (8 * (i & 3));
                            uint32_t bits = 0u;
                            for (int r = 0; r < k_out; ++r) {
                                const int bp = 7 * r;
                                const uint32_t f = __funnelshift_r(w[bp >> 5], w[(bp >> 5) + 1], bp & 31) & 0x7Fu;
                                if (f > 31u) or_status(p.status, OMMX_ST_BAD_GROUP);
                                else bits |= 1u << f;
                            }
                            m2[c] = bits;
                        }
                    }
                    bm2 = make_uint2(m2[0], m2[1]);
                }
                const int nb = KOUT >= 0 ? (KOUT + 1) / 2 : p.nb;
                const uint8_t *ov = gb + o_ov + (hu * 128 + d0) * nb;          // 2*nb bytes, 2-byte aligned
                if (nb == 3) {
                    const uint32_t w0 = reinterpret_cast<const uint16_t *>(ov)[0], w1 = reinterpret_cast<const uint16_t *>(ov)[1],
                                   w2 = reinterpret_cast<const uint16_t *>(ov)[2];
                    st[0] = w0 | ((w1 & 0xFFu) << 16);
                    st[1] = (w1 >> 8) | (w2 << 8);
                } else if (nb == 4) {
                    const uint2 w = *reinterpret_cast<const uint2 *>(ov);
                    st[0] = w.x; st[1] = w.y;
                } else if (nb == 2) {
                    const uint32_t w = *reinterpret_cast<const uint32_t *>(ov);
                    st[0] = w & 0xFFFFu; st[1] = w >> 16;
                } else if (nb > 4) {
                    // 9..16 outliers: the two channels' streams are 2*nb bytes back to back; read them as
                    // 16-bit pieces into a 128-bit little-endian window and cut it at bit 8*nb
                    uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (i < nb) w[i >> 1] |= (uint32_t) reinterpret_cast<const uint16_t *>(ov)[i] << (16 * (i & 1));
                    const int sh = nb > 4 ? 8 * (nb - 4) : 8;        // 8..32 bits of a stream lie above its first word
                    const uint32_t hmask = sh == 32 ? 0xFFFFFFFFu : ((1u << sh) - 1u);
                    st[0] = w[0]; sth[0] = w[1] & hmask;
                    if (sh == 32) { st[1] = w[2]; sth[1] = w[3]; }
                    else { st[1] = __funnelshift_r(w[1], w[2], sh); sth[1] = __funnelshift_r(w[2], w[3], sh) & hmask; }
                } else {
                    const uint32_t w = *reinterpret_cast<const uint16_t *>(ov);
                    st[0] = w & 0xFFu; st[1] = w >> 8;
                }
            }
            if constexpr (PLANES)
                if (splice) {
                    if constexpr (TS < 128) code_bit_planes(smem_u32(k_hi) + swz128((uint32_t)(lm_tok * TS + h * 32 + 16 * hf), SWZ), lane, cw);
                    else code_bit_planes(smem_u32(k_hi + lm_tok * TS) + (((h & 3) * 32 + 16 * hf) ^ k_sw ^ (((uint32_t)(lm_tok * TS) >> 3) & SWZ)), lane, cw);
                }
        }
        // Tile `it` of a unit may be written once the MMA warp has read tile it-1.  Decode warps
        // run up to NS groups ahead and the tiles of one unit are built by different warps, so
        // "tile k was read" events rotate over NS barriers per unit (barrier k % NS, phase
        // k / NS): the newest event a waiter can be missing is then always the one it waits
        // for, never an older phase of the same parity.  A unit without a group in this stage goes
        // through the same hand-overs with nothing in them.
        if (it > 0 && !mbar_wait(bar_tempty + 8 * (MAX_STAGES * unit + ring_slot(it - 1, NS)), ring_phase(it - 1, NS), wait_limit)) {
            if (lane == 0) or_status(p.status, OMMX_ST_TIMEOUT);
            return false;
        }
        if (active) {
            // ---- first the rows of factors (K for the code MMAs, V for P.V): the MMA warp
            //      starts on them while the deltas are scattered ----
            uint8_t *row = tile + ROW_KF * DT_STRIDE + 128 * hf + 64 * (da >> 1) + 16 * dj + 8 * (da & 1) + 2 * dh;
            *reinterpret_cast<uint16_t *>(row) = (uint16_t)kf;
            *reinterpret_cast<uint16_t *>(row + 4) = (uint16_t)(kf >> 16);
            if (hf == 0) {
                uint8_t *at = tile + (ROW_VF + (it & 1)) * DT_STRIDE + 16 * ((lane >> 1) & 3) + 8 * (lane >> 4) + 4 * ((lane >> 3) & 1) + 2 * (lane & 1);
                *reinterpret_cast<uint16_t *>(at) = (uint16_t)f02;
                *reinterpret_cast<uint16_t *>(at + 64) = (uint16_t)f13;
                *reinterpret_cast<uint16_t *>(at + 128) = (uint16_t)(f02 >> 16);
                *reinterpret_cast<uint16_t *>(at + 192) = (uint16_t)(f13 >> 16);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_trows + 8 * unit);
            // ---- then the outlier deltas of this half's columns ----
            if (splice) {
                // clear this half's columns of token rows 0..31 (128 bytes per row)
#pragma unroll
                for (int k2 = 0; k2 < 8; ++k2)
                    *reinterpret_cast<uint4 *>(tile + (4 * k2 + (lane >> 3)) * DT_STRIDE + 128 * hf + 16 * (lane & 7)) = make_uint4(0, 0, 0, 0);
                __syncwarp();                                        // the cleared rows before any delta lands in them
                const uint32_t k_lo = (uint32_t)((h & 3) * 32 + (d0 >> 2)) ^ k_sw;
                auto code_byte = [&](uint32_t pz) -> uint32_t {
                    if constexpr (TS < 128) return k_hi[swz128(pz * TS + k_lo, SWZ)];
                    return k_hi[pz * TS + (k_lo ^ (((pz * TS) >> 3) & SWZ))];
                };
                const uint32_t colp = smem_u32(tile) + 128 * hf + 32 * da + 4 * dj + 2 * dh;
                uint32_t bmv[2] = {bm2.x, bm2.y};
                float scale[2], lvlA[2], offs[2];                // delta of an outlier: lvl * lvlA + offs - code * scale
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    scale[c] = __uint_as_float((uint32_t)(max((int)(int8_t)(e2 >> (8 * c)), -126) + 127) << 23);
                    const float zp = __uint_as_float(c ? z2 & 0xFFFF0000u : z2 << 16);
                    lvlA[c] = scale[c];                          // shared map: lvl*s + zp - (code*s + zp)
                    offs[c] = 0.f;
                    if (use_map) {
                        lvlA[c] = __fdividef(1.f, __uint_as_float(c ? ms2 & 0xFFFF0000u : ms2 << 16));
                        offs[c] = __uint_as_float(c ? mc2 & 0xFFFF0000u : mc2 << 16) - zp;
                    }
                }
                if constexpr (KOUT > 0 && KOUT % 2 == 0) {
                    // a bitmask that disagrees with the value stream: reported, no deltas for that channel
                    const bool bad0 = __popc(bmv[0]) != KOUT, bad1 = __popc(bmv[1]) != KOUT;
                    if (__any_sync(0xFFFFFFFFu, bad0 || bad1)) {
#pragma unroll
                        for (int c = 0; c < 2; ++c)
                            if (c ? bad1 : bad0) {
                                or_status(p.status, OMMX_ST_BAD_GROUP);
                                bmv[c] = (1u << KOUT) - 1u;
                                scale[c] = lvlA[c] = offs[c] = 0.f;
                            }
                    }
                }
                if constexpr (PLANES) {
                    // both channels side by side: two bit walks in flight
#pragma unroll
                    for (int r = KOUT - 2; r >= 0; r -= 2)
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            const uint32_t nib = r < 8 ? (r & 4 ? st[c] >> 16 : st[c]) : (r & 4 ? sth[c] >> 16 : sth[c]);
                            const uint32_t lv = __byte_perm(fp4_levels_hi(nib), 0u, r & 2 ? 0x3424u : 0x1404u);
                            const float2 lvf = __half22float2(*reinterpret_cast<const __half2 *>(&lv));
                            const uint32_t p1 = top_bit(bmv[c]), m1 = 1u << p1;
                            bmv[c] ^= m1;
                            const uint32_t p0 = top_bit(bmv[c]), m0 = 1u << p0;
                            bmv[c] ^= m0;
                            float x0 = fmaf(lvf.x, lvlA[c], offs[c]), x1 = fmaf(lvf.y, lvlA[c], offs[c]);
                            sub_if_bit(x0, cw[2 * c], m0, scale[c]);
                            sub_if_bit(x1, cw[2 * c], m1, scale[c]);
                            sub_if_bit(x0, cw[2 * c + 1], m0, 2.f * scale[c]);
                            sub_if_bit(x1, cw[2 * c + 1], m1, 2.f * scale[c]);
                            sts_u16x2(colp + 16 * c + p0 * DT_STRIDE, colp + 16 * c + p1 * DT_STRIDE, pack_bf16x2(x0, x1));
                        }
                } else {
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    uint32_t bits = bmv[c];
                    const float sc = scale[c], A = lvlA[c], Bc = offs[c];
                    const uint32_t stream = st[c], stream_hi = sth[c];
                    (void)stream_hi;
                    const int fsh = 2 * ((d0 & 3) + c);          // bit position of the channel's code in its byte
                    const uint32_t col = colp + 16 * c;
                    if constexpr (KOUT > 0 && KOUT % 2 == 0) {
                        // The code enters as the fraction of 1 + code/4, whose bits an AND and an OR make, so that 4 * sc moves to
                        // the constant: lvl * A + (Bc + 4 sc) - (1 + code/4) * 4 sc.
                        const float Bq = fmaf(4.f, sc, Bc), Sq = -4.f * sc;
                        const int sh = 21 - fsh;                 // moves the code to the top of the mantissa
                        // Two passes: all gathers (bit walk, base-code byte) first, then the arithmetic and the
                        // stores.  In one pass every load would have to follow the previous outlier's store in
                        // program order (shared memory may alias), i.e. KOUT load round trips in a row.
                        uint32_t pzs[KOUT], cbs[KOUT];
#pragma unroll
                        for (int r = KOUT - 1; r >= 0; --r) {
                            const uint32_t pz = top_bit(bits);
                            bits ^= 1u << pz;
                            pzs[r] = pz;
                            cbs[r] = code_byte(pz);
                        }
#pragma unroll
                        for (int r = 0; r < KOUT; r += 2) {
                            const uint32_t nib = r < 8 ? (r & 4 ? stream >> 16 : stream) : (r & 4 ? stream_hi >> 16 : stream_hi);
                            const uint32_t lv = __byte_perm(fp4_levels_hi(nib), 0u, r & 2 ? 0x3424u : 0x1404u);
                            const float2 lvf = __half22float2(*reinterpret_cast<const __half2 *>(&lv));
                            const float v0 = __uint_as_float(((cbs[r] << sh) & 0x600000u) | 0x3F800000u);
                            const float v1 = __uint_as_float(((cbs[r + 1] << sh) & 0x600000u) | 0x3F800000u);
                            sts_u16x2(col + pzs[r] * DT_STRIDE, col + pzs[r + 1] * DT_STRIDE,
                                      pack_bf16x2(fmaf(v0, Sq, fmaf(lvf.x, A, Bq)), fmaf(v1, Sq, fmaf(lvf.y, A, Bq))));
                        }
                    } else {
                        // any other k: one pass at run time
                        int r = __popc(bits) - 1;
                        while (bits) {
                            const uint32_t pz = top_bit(bits);
                            bits ^= 1u << pz;
                            const uint32_t nib = ((r < 8 ? stream : stream_hi) >> (4 * (r & 7))) & 0xFu;
                            --r;
                            const float cf = (float)((code_byte(pz) >> fsh) & 3u);
                            const float X = fmaf(cf, -sc, fmaf(s_lut[nib], A, Bc));
                            asm volatile("st.shared.b16 [%0], %1;" ::"r"(col + pz * DT_STRIDE), "h"((uint16_t)pack_bf16x2(X, X)) : "memory");
                        }
                    }
                }
                }
            }
        } else if (lane == 0) {
            mbar_arrive(bar_trows + 8 * unit);
        }
        __syncwarp();
        if (lane == 0) {
            mbar_arrive(bar_tfull + 8 * unit);
            mbar_arrive(bar_empty + 8 * s);
        }
        return true;
    };

    bool producer_alive = true;
    auto produce = [&]() __attribute__((always_inline)) {
        const int pw = warp - PRODUCER_WARP;
        const uint32_t full_bytes = stage_bytes_of(pc, 0, true, lane * NPW + pw, 32 * NPW);   // this warp's share of a stage of whole groups
        for (int it = 1;; ++it) {
            bool more = true;
            while (it >= pc.it1 && (more = step_piece())) {}            // a shared piece may hold nothing for this CTA
            if (!more) break;
            lookup_stage(pc, it, NPW, pw);
            const uint32_t bytes = whole_stage(pc, it) ? full_bytes : stage_bytes_of(pc, it, false, lane * NPW + pw, 32 * NPW);
            // the first NS fills find their slots fresh
            if (it >= NS && !mbar_wait(bar_empty + 8 * ring_slot(it, NS), ring_phase(it, NS) ^ 1, wait_limit)) {
                if (lane == 0) or_status(p.status, OMMX_ST_TIMEOUT);
                producer_alive = false;
                break;
            }
            issue_stage(pc, it, NPW, pw, true, bytes);      // a share may hold nothing of a short stage: its announcement still counts
        }
    };

    // ---- roles; each branch resizes its warpgroups' register budget and never rejoins.  What needs no earlier kernel is done before the
    //      wait for it: clearing the tiles, the decode warps' registers (both
    //      stages in a graph: 1K 10.35 -> 9.3 us, 4K 12.5 -> 11.6, 16K 19.5 -> 18.5, 64K 41.6 -> 41.0; with the MMA warps' registers ahead
    //      of it too 11.8 and 41.1, 8 x 32K 136.4 -> 137.3).  The wide layout's producers start the pieces first, which 24
    //      registers do not hold, and its MMA warps need what they give back. ----
    if constexpr (WIDE)
        if (warp >= PRODUCER_WARP) {
            const ShareDivisors by = share_divisors(p.grid, p.S);
            wait_for_earlier_kernels();
            start_pieces(by);
            const bool any = pieces_listed();
            asm volatile("setmaxnreg.dec.sync.aligned.u32 " OMMX_REGS_PRODUCER ";");
            if (any) produce();
            return;
        }
    if (warp >= NCW) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 " OMMX_REGS_DECODE ";");
        if constexpr (WIDE) {
            wait_for_earlier_kernels();
        } else {
            const ShareDivisors by = share_divisors(p.grid, p.S);
            wait_for_earlier_kernels();
            if (warp >= FILL_WARP) start_pieces(by);
        }
        if (!pieces_listed()) return;
        // Narrow layout: with every stage on its way the producer has nothing left to do, while the 15 decode warps share
        // 16 items per iteration: it joins them below for the very last item, so that the last iteration's 16 halves are
        // built side by side.
        if (!WIDE && warp == PRODUCER_WARP) produce();
    // MMA warp w owns unit w = (group-in-stage, kv head) and its softmax state.  The decode warps are
    // stateless: work item number n goes to decode warp n % NDW (narrow layout: except the last one, the producer's).
    {
        // =========================== decode warps (narrow layout: and the producer, once it is done) ===========================
        const int dw = warp - NCW;
        const bool is_producer = !WIDE && warp == PRODUCER_WARP;
        if (is_producer && (!producer_alive || pc.more || (CLUSTER && pc.it0 == pc.it1))) return;
        // the producer takes the very last item, when this CTA's pieces end with one that is known to be the last
        for (int n = is_producer ? pc.it1 * 2 * NCW - 1 : dw;; n += NDW) {
            const int it = n / (2 * NCW);
            bool more = true;
            while (it >= pc.it1 && (more = step_piece())) {}
            if (!more || (!WIDE && !is_producer && !pc.more && n == pc.it1 * 2 * NCW - 1) || !decode_item(pc, n)) break;
        }
        // an exponent that the factors cannot hold was clamped
        if ((int)(e_max & 0xFFFFu) > E_TOP || (int)(e_max >> 16) > E_TOP) or_status(p.status, OMMX_ST_SCALE_RANGE);
        return;
    }
    }

    // =========================== MMA warps ===========================
    wait_for_earlier_kernels();
    const bool any = pieces_listed();
    asm volatile("setmaxnreg.inc.sync.aligned.u32 " OMMX_REGS_MMA ";");
    if (!any) return;
    const int unit = warp;
    const int h = unit % H, gsel = unit / H;
    const uint8_t *tile = s_tiles + unit * DT_BYTES;
    const uint32_t tile_s = smem_u32(tile);
    // Column n = g of every MMA is query head g of this kv head.  Columns past the last head repeat head 0; nobody reads them.
    const bool head_ok = g < p.gqa;
    // per-lane fragment addresses inside the sidecar tile
    const uint32_t a_delta = tile_s + ((lane & 7) + 8 * ((lane >> 3) & 1)) * DT_STRIDE + 16 * (lane >> 4);
    const uint8_t *p_kf = tile + ROW_KF * DT_STRIDE + 16 * j;       // 16-byte piece q2 of lane group j at 64 q2 + 16 j: one line for all four
    // V codes: row r of a 16x16 byte matrix is token sigma(r) = 2 (r / 4) + (r / 2) % 2 + 8 (r % 2) of its 16, so that the four
    // bytes a lane receives are tokens 2j, 8 + 2j, 2j + 1, 9 + 2j: bytes 0 and 2 sit in the two halves of a register as they
    // are, bytes 1 and 3 after a shift.
    const uint32_t v_off = swz128((uint32_t)((2 * ((lane & 15) >> 2) + ((lane >> 1) & 1) + 8 * (lane & 1)) * TS + h * 32 + 16 * (lane >> 4)), SWZ);
    static_assert(SWZ == 0 || (16 * TS) % 1024 == 0, "the second half of the tokens has the same swizzle");
    // V zero-points come out of the plane as an A operand by a transposed load: two heads' four of a token are one 16-byte row
    constexpr int ZROW = H > 1 ? 4 : 0;                             // rows of the odd head
    const int zr = ZROW * (h & 1);
    const bool do_k = !(abl & ABL_NO_K), do_v = !(abl & ABL_NO_V);
    const bool has_delta = !(k_out == 0 || no_outlier);

    constexpr bool keep_last = GS > 1 || CLUSTER;                    // a piece's last tile serves to exchange states before it is handed back
    bool gave_up = false;                        // a wait ran out: no more groups, but every piece still goes through its epilogue
    do {
    // B fragments of q, bf16.  QR: raw, registers 4v..4v+3 hold channels 32v + 8j .. + 7 (zero-point MMAs).  QP: q * sm_scale
    // rounded, register r = 8w + i holds channels (64w + 16j + i, + 8), the pair a code word yields in one AND (code and delta MMAs).
    uint32_t QR[16], QP[16];
    {
        const uint16_t *qrow = reinterpret_cast<const uint16_t *>(p.q + (int64_t)pc.b * p.q_sb + (int64_t)(h * p.gqa + (head_ok ? g : 0)) * p.q_sh);
        auto eight = [&](const uint16_t *q8, uint32_t (&w)[4]) __attribute__((always_inline)) {
            if (p.q_vec_ok) {
                const uint4 t = __ldg(reinterpret_cast<const uint4 *>(q8));
                w[0] = t.x; w[1] = t.y; w[2] = t.z; w[3] = t.w;
            } else {
#pragma unroll
                for (int v = 0; v < 4; ++v) w[v] = (uint32_t)__ldg(q8 + 2 * v) | ((uint32_t)__ldg(q8 + 2 * v + 1) << 16);
            }
        };
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            uint32_t w[4];
            eight(qrow + 32 * v + 8 * j, w);
#pragma unroll
            for (int i = 0; i < 4; ++i) QR[4 * v + i] = w[i];
        }
        auto scaled = [&](uint32_t b16) { return bf16_bits_to_f32(b16 & 0xFFFFu) * p.sm_scale; };
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            uint32_t lo[4], hi[4];
            eight(qrow + 64 * w + 16 * j, lo);
            eight(qrow + 64 * w + 16 * j + 8, hi);
#pragma unroll
            for (int i = 0; i < 8; ++i)
                QP[8 * w + i] = pack_bf16x2(scaled(lo[i >> 1] >> (16 * (i & 1))), scaled(hi[i >> 1] >> (16 * (i & 1))));
        }
    }
    // ---- online softmax state of heads 2j and 2j+1 (the two columns this lane holds) ----
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
    // acc[2*cg + u]: rows = channels 32cg + 4g + u (regs 0,1) and 32cg + 4g + 2 + u (regs 2,3), columns = heads
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i) { acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f; }
    float accz[4] = {0.f, 0.f, 0.f, 0.f};        // rows = V scale groups (from row zr): sum_t vz[t][cg] * P[t][head]

    for (int it = pc.it0; it < pc.it1 && !gave_up; ++it) {
        const int s = ring_slot(it, NS);
        const uint32_t ph = ring_phase(it, NS);
        const int lg = (it - pc.it0) * GS + gsel;                    // local group of this warp
        const bool active = lg < pc.ng && !(abl & ABL_NO_COMPUTE);
        if (!mbar_wait(bar_full + 8 * s, ph, wait_limit)) {
            gave_up = true;
            break;
        }
        if (active) {
            uint8_t *gb = s_stage + (size_t)s * stage_bytes + (GATHER ? 0 : (size_t)gsel * gb_bytes);
            const uint32_t rows_at = GATHER ? gsel * H * 1024 : 0;        // token rows of the group in either code plane
            const uint32_t v_addr = smem_u32(gb + o_vm) + rows_at + v_off;  // v_main region of the group (1 KB aligned)

            // ======================= logits =======================
            // code words of this lane's four token rows (tokens 8*nt + g), channels 16j..16j+15 of either half
            uint32_t kw[2][4] = {};
            if (do_k)
#pragma unroll
                for (int w = 0; w < 2; ++w)
                    ldsm_x4(smem_u32(gb) + rows_at + swz128((uint32_t)(lane * TS + h * 32 + 16 * w), SWZ), kw[w][0], kw[w][1], kw[w][2], kw[w][3]);
            // The unit's sidecar tile arrives in two steps: first the rows of factors, then the outlier
            // deltas.  The code MMAs run on the first, while the decode warps still scatter the deltas.
            if (!mbar_wait(bar_trows + 8 * unit, (uint32_t)it & 1u, wait_limit)) {
                gave_up = true;
                break;
            }
            float Sc[2][4], Sd[2][4];
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) { Sc[mt][0] = Sc[mt][1] = Sc[mt][2] = Sc[mt][3] = 0.f; Sd[mt][0] = Sd[mt][1] = Sd[mt][2] = Sd[mt][3] = 0.f; }
            // Two accumulators take turns, so that neighbours in the instruction stream never wait on each other
            // (the asm statements keep their order, so the order written here is the order issued).
#pragma unroll
            for (int q2 = 0; q2 < 4; ++q2) {
                const uint4 f = *reinterpret_cast<const uint4 *>(p_kf + 64 * q2);      // two k-steps' factor pairs
#pragma unroll
                for (int q = 2 * q2; q < 2 * q2 + 2; ++q) {
                    const int wi = q >> 2, i0 = 2 * (q & 3);
                    const uint32_t b0 = hmul2_bf16(QP[2 * q], q & 1 ? f.z : f.x), b1 = hmul2_bf16(QP[2 * q + 1], q & 1 ? f.w : f.y);
#pragma unroll
                    for (int mt = 0; mt < 2; ++mt) {
                        const uint32_t wlo = kw[wi][2 * mt], whi = kw[wi][2 * mt + 1];
                        mma_bf16(Sc[mt], code_pair_bf16(wlo, i0), code_pair_bf16(whi, i0), code_pair_bf16(wlo, i0 + 1), code_pair_bf16(whi, i0 + 1), b0, b1);
                    }
                }
            }
            // q.zp of heads 2j and 2j+1: exact bf16 products of the raw query with the zero-points, summed in fp32.  It needs no tile, so
            // it stands where this warp may have to wait for the deltas.  The eight zero-points a lane loads stand in an A operand as
            // they come, rows 0-7 holding words 0 and 2, rows 8-15 words 1 and 3: with the query's words 0 and 2 the first rows are
            // of use, with 1 and 3 the others.
            float Z0[4] = {0.f, 0.f, 0.f, 0.f}, Z1[4] = {0.f, 0.f, 0.f, 0.f};
            {
                const uint8_t *zrow = gb + o_kz + (GATHER ? unit : h) * 256 + 16 * j;
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    const uint4 z = *reinterpret_cast<const uint4 *>(zrow + 64 * v);
                    mma_bf16(Z0, z.x, z.y, z.z, z.w, QR[4 * v], QR[4 * v + 2]);
                    mma_bf16(Z1, z.x, z.y, z.z, z.w, QR[4 * v + 1], QR[4 * v + 3]);
                }
            }
            const float Sz[2] = {(Z0[0] + Z1[2]) * p.sm_scale, (Z0[1] + Z1[3]) * p.sm_scale};
            if (has_delta) {
                if (!mbar_wait(bar_tfull + 8 * unit, (uint32_t)it & 1u, wait_limit)) {
                    gave_up = true;
                    break;
                }
                uint32_t d0f[4], d1f[4];                         // delta fragments of m-tile 0 / 1
                ldsm_x4(a_delta, d0f[0], d0f[1], d0f[2], d0f[3]);
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    ldsm_x4(a_delta + 16 * DT_STRIDE + 32 * q, d1f[0], d1f[1], d1f[2], d1f[3]);
                    mma_bf16(Sd[0], d0f[0], d0f[1], d0f[2], d0f[3], QP[2 * q], QP[2 * q + 1]);
                    if (q < 7) ldsm_x4(a_delta + 32 * (q + 1), d0f[0], d0f[1], d0f[2], d0f[3]);
                    mma_bf16(Sd[1], d1f[0], d1f[1], d1f[2], d1f[3], QP[2 * q], QP[2 * q + 1]);
                }
            }
            __syncwarp();
            // the next tile may be built (where warps merge below, they do it in their tiles: not before that)
            if (lane == 0 && (!keep_last || it + 1 < pc.it1)) mbar_arrive(bar_tempty + 8 * (MAX_STAGES * unit + ring_slot(it, NS)));

            // ======================= online softmax =======================
            // x[mt][r]: token 16mt + g + 8(r>>1), head 2j + (r&1)
            float x[2][4];
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int r = 0; r < 4; ++r) x[mt][r] = fmaf(Sc[mt][r], KF_UNDO, Sd[mt][r] + Sz[r & 1]);
            if (!PLAIN && p.logit_cap > 0.f) {
#pragma unroll
                for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                    for (int r = 0; r < 4; ++r) x[mt][r] = p.logit_cap * tanhf(x[mt][r] / p.logit_cap);
            }
            const int tok_base = 32 * lg;
            if (tok_base + 32 > pc.ntok) {
#pragma unroll
                for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        if (tok_base + 16 * mt + g + 8 * (r >> 1) >= pc.ntok) x[mt][r] = -INFINITY;
            }
            // The reference maximum follows only when a logit is more than LAG ahead of it, so that most units need neither the
            // maximum over the lanes nor a rescaled accumulator.  P may then be up to e^LAG, which the largest V factor just allows;
            // against a maximum LAG further up, small P would lose bits (errors against 64-bit attention 2 to 4 % larger).
            bool ahead = false;
            float mloc[2];
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                mloc[hh] = fmaxf(fmaxf(x[0][hh], x[0][2 + hh]), fmaxf(x[1][hh], x[1][2 + hh]));
                ahead = ahead || mloc[hh] > m_run[hh] + LAG;
            }
            if (__any_sync(0xFFFFFFFFu, ahead)) {
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    mloc[hh] = fmaxf(mloc[hh], __shfl_xor_sync(0xFFFFFFFFu, mloc[hh], 4));
                    mloc[hh] = fmaxf(mloc[hh], __shfl_xor_sync(0xFFFFFFFFu, mloc[hh], 8));
                    mloc[hh] = fmaxf(mloc[hh], __shfl_xor_sync(0xFFFFFFFFu, mloc[hh], 16));
                    const float m_new = fmaxf(m_run[hh], mloc[hh]);
                    const float m_use = (m_new == -INFINITY) ? 0.f : m_new;
                    const float corr = fast_exp2((m_run[hh] - m_use) * LOG2E);   // m_run = -inf -> 0
                    m_run[hh] = m_new;
                    l_run[hh] *= corr;
#pragma unroll
                    for (int i = 0; i < 8; ++i) { acc[i][hh] *= corr; acc[i][2 + hh] *= corr; }
                    accz[hh] *= corr;
                }
            }
            const float mneg[2] = {m_run[0] == -INFINITY ? 0.f : -m_run[0] * LOG2E, m_run[1] == -INFINITY ? 0.f : -m_run[1] * LOG2E};
            float pr[2][4];
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int r = 0; r < 4; ++r) pr[mt][r] = fast_exp2(fmaf(x[mt][r], LOG2E, mneg[r & 1]));
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) l_run[hh] += (pr[0][hh] + pr[0][2 + hh]) + (pr[1][hh] + pr[1][2 + hh]);   // this lane's tokens only
            // P^T as B fragments: transpose each 8x8 (token, head) block; T[ks][b] = tokens 16ks + 8b + 2j, +1 of head g
            uint32_t T[2][2];
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
                T[mt][0] = movmatrix_trans(pack_f16x2(pr[mt][0], pr[mt][1]));
                T[mt][1] = movmatrix_trans(pack_f16x2(pr[mt][2], pr[mt][3]));
            }

            // ======================= P.V =======================
            if (do_v) {
                const int copy = it & 1;
                uint32_t VF[16];                                     // factor pairs, index 4cg + 2ks + b
                {
                    const uint8_t *p_vf = tile + (ROW_VF + copy) * DT_STRIDE + 16 * j;
#pragma unroll
                    for (int v = 0; v < 4; ++v) {
                        const uint4 t = *reinterpret_cast<const uint4 *>(p_vf + 64 * v);
                        VF[4 * v] = t.x; VF[4 * v + 1] = t.y; VF[4 * v + 2] = t.z; VF[4 * v + 3] = t.w;
                    }
                }
                // zero-points: z[m] = tokens 8m + 2j, + 1 of row g
                uint32_t z[4];
                if constexpr (H > 1) {
                    ldsm_x4_trans(smem_u32(gb + o_vz + (GATHER ? gsel * H * 256 : 0) + (lane * H + (h & ~1)) * 8), z[0], z[1], z[2], z[3]);
                } else {
#pragma unroll
                    for (int m = 0; m < 4; ++m) {
                        const uint16_t *vz = reinterpret_cast<const uint16_t *>(gb + o_vz + (GATHER ? gsel * H * 256 : 0) + (8 * m + 2 * j) * 8) + (g & 3);
                        z[m] = g < 4 ? (uint32_t)vz[0] | ((uint32_t)vz[4] << 16) : 0u;
                    }
                }
                if (tok_base + 32 > pc.ntok) {                                     // what no token of this sequence wrote may be anything
#pragma unroll
                    for (int m = 0; m < 4; ++m) {
                        if (8 * m + 2 * j + tok_base >= pc.ntok) z[m] = 0u;
                        else if (8 * m + 2 * j + 1 + tok_base >= pc.ntok) z[m] &= 0xFFFFu;
                    }
                }
#pragma unroll
                for (int ks = 0; ks < 2; ++ks) {
                    uint32_t vc[4];                                  // by scale group: channels 32cg + 4g .. + 3 of four tokens, a byte each
                    ldsm_b8_trans_x2(v_addr + 16 * TS * ks, vc);
#pragma unroll
                    for (int cg = 0; cg < 4; ++cg) {
                        const uint32_t w01 = vc[cg], w89 = vc[cg] >> 8;
                        const uint32_t pb0 = hmul2_f16(T[ks][0], VF[4 * cg + 2 * ks]), pb1 = hmul2_f16(T[ks][1], VF[4 * cg + 2 * ks + 1]);
#pragma unroll
                        for (int u = 0; u < 2; ++u)
                            mma_f16(acc[2 * cg + u], w01 & (0x00030003u << (2 * u)), w01 & (0x00030003u << (2 * u + 4)),
                                    w89 & (0x00030003u << (2 * u)), w89 & (0x00030003u << (2 * u + 4)), pb0, pb1);
                    }
                    const uint32_t z0 = z[2 * ks], z1 = z[2 * ks + 1];
                    mma_f16(accz, pack_f16x2_sat(bf16_bits_to_f32(z0), __uint_as_float(z0 & 0xFFFF0000u)), 0u,
                            pack_f16x2_sat(bf16_bits_to_f32(z1), __uint_as_float(z1 & 0xFFFF0000u)), 0u, T[ks][0], T[ks][1]);
                }
            }
        } else {
            if (!mbar_wait(bar_trows + 8 * unit, (uint32_t)it & 1u, wait_limit)) {
                gave_up = true;
                break;
            }
            if (lane == 0 && (!keep_last || it + 1 < pc.it1)) mbar_arrive(bar_tempty + 8 * (MAX_STAGES * unit + ring_slot(it, NS)));
        }
        // release the stage
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_empty + 8 * s);
    }
    if (gave_up) {
        if (lane == 0) or_status(p.status, OMMX_ST_TIMEOUT);
        m_run[0] = m_run[1] = -INFINITY; l_run[0] = l_run[1] = 0.f;
    }

    // ---- epilogue: this lane holds 16 channels of heads 2j and 2j+1; merge warps that share a head ----
    float l_tot[2];
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
        float l = l_run[hh];
        l += __shfl_xor_sync(0xFFFFFFFFu, l, 4);
        l += __shfl_xor_sync(0xFFFFFFFFu, l, 8);
        l += __shfl_xor_sync(0xFFFFFFFFu, l, 16);
        l_tot[hh] = l;
    }
    // outv[hh][4cg + c]: channel 32cg + 4g + c of head 2j + hh, un-normalised
    float outv[2][16];
#pragma unroll
    for (int cg = 0; cg < 4; ++cg) {
        const float bz0 = __shfl_sync(0xFFFFFFFFu, accz[0], 4 * (zr + cg) + j);
        const float bz1 = __shfl_sync(0xFFFFFFFFu, accz[1], 4 * (zr + cg) + j);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int u = c & 1, v = c >> 1;
            const float f = 1048576.f / (float)(1 << (2 * c));       // 2^(24 - FBIAS) * 4^-slot
            outv[0][4 * cg + c] = fmaf(acc[2 * cg + u][2 * v], f, bz0);
            outv[1][4 * cg + c] = fmaf(acc[2 * cg + u][2 * v + 1], f, bz1);
        }
    }

    // softmax state (m2, l2, un-normalised rows `other(i)`) into this warp's
    auto merge_state = [&](auto other) __attribute__((always_inline)) {
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            const float m2 = other(hh), l2 = other(2 + hh);
            const float mn = fmaxf(m_run[hh], m2);
            const float mu = (mn == -INFINITY) ? 0.f : mn;
            const float c1 = fast_exp2((m_run[hh] - mu) * LOG2E), c2 = fast_exp2((m2 - mu) * LOG2E);
            l_tot[hh] = l_tot[hh] * c1 + l2 * c2;
#pragma unroll
            for (int i = 0; i < 16; ++i) outv[hh][i] = outv[hh][i] * c1 + other(4 + 16 * hh + i) * c2;
            m_run[hh] = mn;
        }
    };
    auto store_state = [&]() __attribute__((always_inline)) {
        float *my = reinterpret_cast<float *>(s_tiles + unit * DT_BYTES) + lane;
        my[0] = m_run[0]; my[32] = m_run[1]; my[64] = l_tot[0]; my[96] = l_tot[1];
#pragma unroll
        for (int i = 0; i < 16; ++i) { my[32 * (4 + i)] = outv[0][i]; my[32 * (20 + i)] = outv[1][i]; }
    };
    // Several groups per stage (fewer than 8 local kv heads): the warps that share a head merge, each through the delta rows
    // of its own tile, which nobody builds again before it is handed back below.  With 8 heads every warp owns its head.
    static_assert(32 * 36 * 4 <= 32 * DT_STRIDE, "the merge fits the delta rows of a tile");
    const bool mine = !CLUSTER || pc.it0 < pc.it1;                   // this CTA had groups of the piece
    constexpr bool TOGETHER = GS > 2 && !CLUSTER;
    if constexpr (TOGETHER) {
        // All at once: of the head's 32 values a lane holds, warp gsel takes 32 / GS from every warp's tile and writes them out (one
        // warp that merged the others one by one, both stages: 8 x 32K x 1 head 30.6 -> 29.6 us, 8K 11.4 -> 10.3; 128K x 2 heads
        // 28.1 -> 27.4, 4K 10.8 -> 10.3).  Of two warps (four heads) one merges the other's: 32K 19.5 us, together 19.8.
        // In clusters one warp merges too: it holds the whole state that the CTAs exchange.  Side by side there is not tried.
        store_state();
        asm volatile("bar.sync 3, %0;" ::"n"(NCW * 32) : "memory");
        constexpr int NCG = 8 / GS;
        const int hh = 2 * gsel / GS, cg0 = gsel % (GS / 2) * NCG, head = 2 * j + hh;
        const float *states = reinterpret_cast<const float *>(s_tiles + h * DT_BYTES) + lane;
        constexpr int NEXT = H * DT_BYTES / 4;                      // floats from one warp's state to the next of the same head
        float m = -INFINITY, l = 0.f, c[GS], sum[4 * NCG] = {};
#pragma unroll
        for (int o = 0; o < GS; ++o) m = fmaxf(m, c[o] = states[o * NEXT + 32 * hh]);
        const float mu = m == -INFINITY ? 0.f : m;
#pragma unroll
        for (int o = 0; o < GS; ++o) {
            c[o] = fast_exp2((c[o] - mu) * LOG2E);
            l += c[o] * states[o * NEXT + 32 * (2 + hh)];
#pragma unroll
            for (int i = 0; i < 4 * NCG; ++i) sum[i] += c[o] * states[o * NEXT + 32 * (4 + 16 * hh + 4 * cg0 + i)];
        }
        if (head < p.gqa) {
            const float inv = l > 0.f ? 1.f / l : 0.f;
            float *dst = p.al + (int64_t)pc.b * p.al_sb + (int64_t)(h * p.gqa + head) * p.al_sh + (int64_t)pc.slot * p.al_ss;
#pragma unroll
            for (int i = 0; i < 4 * NCG; ++i) dst[32 * (cg0 + i / 4) + 4 * g + i % 4] = sum[i] * inv;
            if (g == 0 && cg0 == 0) dst[HD] = l > 0.f ? m + logf(l) : -INFINITY;
        }
        asm volatile("bar.sync 3, %0;" ::"n"(NCW * 32) : "memory");
    } else if (GS > 1 && mine) {
        if (gsel > 0) store_state();
        asm volatile("bar.sync 3, %0;" ::"n"(NCW * 32) : "memory");
        if (gsel == 0) {
#pragma unroll 1
            for (int o = 1; o < GS; ++o) {
                const float *ot = reinterpret_cast<const float *>(s_tiles + (o * H + h) * DT_BYTES) + lane;
                merge_state([&](int i) { return ot[32 * i]; });
            }
        }
        asm volatile("bar.sync 3, %0;" ::"n"(NCW * 32) : "memory");
    }
    bool write = gsel == 0 && !TOGETHER;
    if constexpr (CLUSTER)
    if (gsel == 0 && *s_ctas > 1) {
        // the CTAs that share the piece: head h is merged by CTA h % n_ctas
        const int n_ctas = *s_ctas, rank = cluster_rank(), to = h % n_ctas;
        const uint32_t there = s_there + 8 * h;
        write = rank == to;
        // A warp that has given up takes no further part: it neither waits nor arrives, so no barrier runs ahead of those who still
        // do, each of which gives up once in turn, and the launch ends within two or three limits.  With further waits it could take
        // fifteen, with arrivals but no waits, whose phases alias, six (a model of the barriers over random pieces).  The lanes agree on
        // it, whichever of them saw the clock run out.
        auto wait_peers = [&](uint32_t bar) __attribute__((always_inline)) {
            if (__all_sync(0xFFFFFFFFu, mbar_wait_peers(bar, (uint32_t)pi & 1u, wait_limit))) return;
            gave_up = true;
            if (lane == 0) or_status(p.status, OMMX_ST_TIMEOUT);
        };
        if (gave_up) {
        } else if (!write) {
            if (mine) store_state();
            if (lane == 0) asm volatile("st.shared.u32 [%0], %1;" ::"r"(there), "r"((uint32_t)mine) : "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_peer(peer_smem(bar_handed + 8 * h, to));
            wait_peers(bar_taken + 8 * h);
        } else {
            wait_peers(bar_handed + 8 * h);
            const uint32_t tile_l = smem_u32(tile) + 4 * lane;
#pragma unroll 1
            for (int o = 1; o < n_ctas && !gave_up; ++o) {           // not all have stored theirs where the wait gave up
                const uint32_t from = (rank + o) % n_ctas;
                if (__float_as_uint(lds_peer(peer_smem(there, from))) == 0u) continue;
                const uint32_t at = peer_smem(tile_l, from);
                merge_state([&](int i) { return lds_peer(at + 128 * i); });
            }
            __syncwarp();
            if (!gave_up && lane < n_ctas && lane != rank) mbar_arrive_peer(peer_smem(bar_taken + 8 * h, lane));
        }
    }
    if (write) {
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            const int head = 2 * j + hh;
            if (head < p.gqa) {
                const float inv = l_tot[hh] > 0.f ? 1.f / l_tot[hh] : 0.f;
                float *dst = p.al + (int64_t)pc.b * p.al_sb + (int64_t)(h * p.gqa + head) * p.al_sh + (int64_t)pc.slot * p.al_ss;
#pragma unroll
                for (int cg = 0; cg < 4; ++cg)
#pragma unroll
                    for (int c = 0; c < 4; ++c) dst[32 * cg + 4 * g + c] = outv[hh][4 * cg + c] * inv;
                if (g == 0) dst[HD] = l_tot[hh] > 0.f ? m_run[hh] + logf(l_tot[hh]) : -INFINITY;
            }
        }
    }
    if (keep_last && mine && lane == 0) mbar_arrive(bar_tempty + 8 * (MAX_STAGES * unit + ring_slot(pc.it1 - 1, NS)));
    } while (step_piece());
    // no CTA leaves while another of its cluster may still read its tiles or arrive on its barriers; warps that left count as arrived
    if constexpr (CLUSTER)
        if (*s_ctas > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Launch as a programmatic dependent of whatever precedes it in the stream: the grid may be placed while that
// kernel drains, and the kernel itself waits (griddepcontrol.wait) before it reads or writes global memory.
template <typename Kernel, typename Params>
static cudaError_t launch_overlapping_previous(Kernel kernel, dim3 grid, int threads, size_t smem, cudaStream_t st, const Params &p, int cluster = 1) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, p);
}

// Lets `kernel` be launched with up to SMEM_LIMIT of dynamic shared memory; `done` holds what has been done on each device.  Always
// the limit, not what the call needs: of two threads whose first calls need different sizes, the smaller could come last.
template <typename Kernel> static int allow_full_smem(Kernel kernel, std::atomic<int> (&done)[MAX_DEVICES], int dev) {
    if (done[dev].load(std::memory_order_acquire) == 0) {
        OMMX_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_LIMIT));
        done[dev].store(1, std::memory_order_release);
    }
    return 0;
}

template <int KOUT, int H, bool PLAIN, bool IDX7, bool CLUSTER>
static int launch_s1(const typename Stage1Form<H, PLAIN>::Params &p, size_t smem, cudaStream_t st) {
    using L = typename Stage1Form<H, PLAIN>::Layout;
    // function attributes belong to (kernel instantiation, device): one entry per device ordinal
    static std::atomic<int> smem_set[MAX_DEVICES];
    static std::atomic<int> regs_state[MAX_DEVICES];   // 0 unknown, 1 enough, 2 too few
    int dev = 0;
    if (int rc = current_device(&dev)) return rc;
    int regs_ok = regs_state[dev].load(std::memory_order_acquire);
    if (regs_ok == 0) {
        cudaFuncAttributes fa;
        OMMX_CUDA_TRY(cudaFuncGetAttributes(&fa, decode_stage1_kernel<KOUT, H, PLAIN, IDX7, CLUSTER>));
        // setmaxnreg.inc must find the registers the other roles gave back
        const int need = NCW * 32 * REGS_MMA + (L::WIDE ? L::NDW * 32 * REGS_DECODE + L::NPW * 32 * REGS_PRODUCER
                                                        : (L::THREADS - NCW * 32) * REGS_DECODE);
        regs_ok = fa.numRegs * L::THREADS >= need ? 1 : 2;
        regs_state[dev].store(regs_ok, std::memory_order_release);
    }
    if (regs_ok != 1) return fail(OMMX_E_CUDA, "stage 1 was compiled with fewer registers than its warp roles need");
    if (int rc = allow_full_smem(decode_stage1_kernel<KOUT, H, PLAIN, IDX7, CLUSTER>, smem_set, dev)) return rc;
    OMMX_CUDA_TRY(launch_overlapping_previous(decode_stage1_kernel<KOUT, H, PLAIN, IDX7, CLUSTER>, dim3(p.grid.ncta), L::THREADS, smem, st, p, p.grid.cluster));
    count_launch();
    return 0;
}
// The tensor maps of a launch: of the code planes by page where that is how they are staged (4 and 8 kv heads), into p, and with `rows` those
// of the planes by row (not of an outlier index whose rows are too long).
int set_plane_maps(S1Params &p, CUtensorMap *rows);

// The form that can exchange states only in launches of clusters, the general form too: in the others its code costs 2 to 6 % (both
// stages, with -> without, 8 kv heads: 4K, k = 3 13.4 -> 12.6 us; 64K, k = 3 44.7 -> 43.5, with a logit cap 53.9 -> 52.6; 70B heads
// 8 x 32K with a logit cap 186.5 -> 183.0, of one kv head 38.2 -> 37.4).
template <int KOUT, int H, bool PLAIN, bool IDX7>
static int launch_s1_form(const S1Params &q, size_t smem, cudaStream_t st) {
    typename Stage1Form<H, PLAIN>::Params p;
    static_cast<S1Params &>(p) = q;
    CUtensorMap *rows = nullptr;
    if constexpr (Stage1Form<H, PLAIN>::GATHER) rows = p.rows;
    if (int rc = set_plane_maps(p, rows)) return rc;
    return p.grid.cluster > 1 ? launch_s1<KOUT, H, PLAIN, IDX7, true>(p, smem, st) : launch_s1<KOUT, H, PLAIN, IDX7, false>(p, smem, st);
}
// The plain form where the recipe and the ring depth are its own, else the general one.
template <int KOUT, int H>
static int launch_s1_forms(const S1Params &p, size_t smem, cudaStream_t st) {
    if constexpr (KOUT >= 0) {
        const bool mapped = !Stage1Form<H, true>::GATHER || (p.num_pages > 0 && p.num_slots > 0);      // an empty plane has no map
        if (p.abl == 0 && (KOUT == 0 || p.use_map) && p.logit_cap <= 0.f && mapped) {
            if (!p.idx7 && p.nstages >= PlainLayout<KOUT, H, false>::STAGES) return launch_s1_form<KOUT, H, true, false>(p, smem, st);
            if constexpr (KOUT > 0)
                if (p.idx7 && p.nstages >= PlainLayout<KOUT, H, true>::STAGES) return launch_s1_form<KOUT, H, true, true>(p, smem, st);
        }
    }
    return launch_s1_form<KOUT, H, false, false>(p, smem, st);
}
// The outlier counts of the serving recipes get the unrolled two-pass splice.
template <int H>
static int launch_s1_heads(const S1Params &p, size_t smem, cudaStream_t st) {
    switch (p.k_out) {
        case 0: return launch_s1_forms<0, H>(p, smem, st);
        case 2: return launch_s1_forms<2, H>(p, smem, st);
        case 4: return launch_s1_forms<4, H>(p, smem, st);
        case 6: return launch_s1_forms<6, H>(p, smem, st);
        case 8: return launch_s1_forms<8, H>(p, smem, st);
        case 12: return launch_s1_forms<12, H>(p, smem, st);
        default: return launch_s1_forms<-1, H>(p, smem, st);
    }
}

// one per translation unit
int launch_stage1_h8(const S1Params &p, size_t smem, cudaStream_t st);
int launch_stage1_h4(const S1Params &p, size_t smem, cudaStream_t st);
int launch_stage1_h2(const S1Params &p, size_t smem, cudaStream_t st);
int launch_stage1_h1(const S1Params &p, size_t smem, cudaStream_t st);

}  // namespace ommx

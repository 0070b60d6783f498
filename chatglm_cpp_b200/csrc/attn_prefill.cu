// Prompt attention on 5th-generation tensor cores (tcgen05 + TMEM) for head_dim 128 (sm_100a).
//
// Covers chatglm.cpp:655-717 for the prompts of a call (n_past == 0, at least kPrefillMinTokens tokens), in two launches for up
// to kPrefillMaxSeq of them:
//   prefill_append_kernel  RoPE on k (:655-656) and the f16 append of the K rows and V^T columns (:668-675);
//   prefill_attn_kernel    RoPE on q, q * 1/sqrt(d) (:686) and flash attention over the cache (:687-717).
// An attention CTA works on TWO 128-row q tiles at a time that read the same K and V^T tiles: the same token rows of two
// q heads of one kv head, or (one q head per kv head) two neighbouring row tiles of a head.  Per 64 tokens (a step) and q tile
// the tensor core has 640 cycles to do (Q K^T: 8 MMAs of 48 cycles, bound by the shared-memory reads of both operands; P V: 4 of
// 64) and the exponential unit 512 (16 per cycle): with one q tile in flight the two alternate, with two they overlap.
//   softmax warps  two groups of four; a thread owns one q row of its group's tile (one tensor-memory lane), so the online
//                  softmax needs no cross-thread reduction.  The scores of a step are released as soon as they are in
//                  registers; the probabilities go back to TENSOR memory and are the A operand of P V there: no shared
//                  memory, no proxy fence.
//   load warp      TMA: K and V^T tiles alternate through one ring (non-multicast, 128-byte swizzle).
//   MMA warps      one per group.  Q K^T of step t + 1 runs while the softmax works on step t, P V of t follows it.  tcgen05.mma
//                  of one thread execute in order: a group that sees its scores of step t knows that P V of t - 2 has landed.
//   q warps        stage the q tiles of the CTA's next unit (CTAs are persistent; units are dealt longest first).
// Measured (B200, 32 q heads, 2 kv heads, causal): an 8192-token prompt alone 491 us, 555 us back to back under the power cap
// (990 TFLOP/s of useful work), against 795 us with one q tile per CTA, probabilities through shared memory and q staged
// through HBM by a kernel of its own.
// A step takes about 1600 cycles; taking a quarter of the exponentials off their unit (a polynomial on the FMA pipe) made it
// slower, because what the softmax warps issue delays the MMA warps, which need about a tenth of the issue slots.
// O stays in tensor memory across KV tiles; a row's O is rescaled there only when its running maximum grows by more than
// 2^8, otherwise the old reference maximum is kept (exact: the same reference enters numerator and denominator).
// Masks (chatglm.cpp:689-707): causal (token t visible to row s iff t <= n_virtual + s; tiles right
// of the diagonal are skipped) or the ChatGLM-6B v1 prefix mask (every row but the last is blocked from the last token).
// Tokens past the attended length: their scores are masked whatever the cache holds there, and the V^T tensor map of a
// sequence ends at its attended length, so TMA fills the rest with zeros.
#include <type_traits>

#include "common.cuh"

namespace cglm {

namespace {

constexpr int kD = 128;
constexpr int kQTile = 128;                   // q rows per tile = TMEM lanes
constexpr int kKvTile = 128;                  // tokens per TMA tile of K or V^T
constexpr int kStep = 64;                     // tokens per softmax step: half a tile
constexpr int kGroupThreads = 128;            // softmax threads per q tile
constexpr int kQWarp = 8;                     // four warps that stage the q tiles of a CTA's next unit
constexpr int kLoadWarp = 12;                 // issues the TMA loads of K and V^T
constexpr int kMmaWarp = 13;                  // kMmaWarp + w issues the MMAs of group w
constexpr int kThreads = 16 * 32;             // (warp 15 idle: register shares are handed out per four warps)
constexpr int kSoftmaxRegs = 168, kOtherRegs = 88;   // 256 x 168 + 256 x 88 = the 65536 registers the CTA is launched with
constexpr int kHalfBytes = 128 * 128;         // one 128-row x 128-byte swizzled half tile (16 KiB)
constexpr int kTileBytes = 2 * kHalfBytes;    // a 128 x 128 f16 operand tile
constexpr int kStages = 5;                    // ring of K and V^T tiles: K(0), V(0), K(1), V(1), ...
constexpr int kTmemCols = 512;                // group w: S at columns 128 w, P buffers at 128 w + 64 and + 96, O at 256 + 128 w
constexpr float kRescaleThreshold = 8.f;      // log2 units a row's maximum may grow before O is rescaled
constexpr float kLog2e = 1.4426950408889634f;
// Reference maximum of a row that has seen no score above -inf (masked tokens, keys that overflowed f16): its exponents are
// ex2(-inf - this) = 0, not NaN.
constexpr float kNoMax = -1.0e30f;

// instruction descriptors of tcgen05.mma.kind::f16: D = f32, A = B = f16, both K-major, M = 128, N = 64 (scores) / 128 (P V)
constexpr uint32_t kIdescS = (1u << 4) | ((64u >> 3) << 17) | ((128u >> 4) << 24);
constexpr uint32_t kIdescO = (1u << 4) | ((128u >> 3) << 17) | ((128u >> 4) << 24);

struct __align__(1024) PrefillSmem {
    uint8_t q[2][kTileBytes];         // A of QK^T per group: [2 d-halves][128 rows][64 d]
    uint8_t kv[kStages][kTileBytes];  // K tile [2 d-halves][128 tokens][64 d] or V^T tile [2 token-halves][128 d][64 tokens]
    uint64_t kv_full[kStages];        // TMA -> MMA: tile landed
    uint64_t kv_empty[kStages];       // tensor core -> TMA: tile has been read by both groups' MMAs
    uint64_t q_full[2];               // q tile of a unit in place (first unit: softmax group, later ones: bulk copy) -> MMA
    uint64_t q_empty[2];              // tensor core -> q warps: the unit's last scores computed
    uint64_t s_full[2];               // tensor core -> softmax group: scores of a step written
    uint64_t s_empty[2];              // softmax group -> MMA: scores are in registers
    uint64_t p_full[2][2];            // softmax group -> MMA: probabilities of a step written, O rescaled if it had to be (per buffer)
    uint64_t o_step[2];               // tensor core -> softmax group: P V of a step accumulated (looked at before a rescale)
    uint64_t o_full[2];               // tensor core -> softmax group: the unit's last P V accumulated
    uint64_t o_empty[2];              // softmax group -> MMA: O of the unit has been read
    uint32_t tmem_base;
    int abort_flag;
};
static_assert(sizeof(PrefillSmem) + 1024 <= 232448, "one prefill CTA must fit the shared memory of an SM");

// Shared-memory matrix descriptor: K-major operand, 128-byte swizzle, 8-row groups 1024 bytes apart.  Its upper word is the
// same for every operand here; an operand `bytes` further on has the lower word + (bytes >> 4).
constexpr uint32_t kDescHi = 64u | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t desc_lo(uint32_t saddr) { return ((saddr & 0x3ffffu) >> 4) | (1u << 16); }
// MMAs and commits of a warp: every lane runs through them and `lead` (one lane's 1) predicates the instruction itself, so that
// the operands are computed in uniform registers; behind a branch on the elected lane each of them was moved there one by one,
// and issuing a 48-cycle MMA took longer than that while the softmax warps kept the schedulers busy.
template <uint32_t kIdesc, bool kAccumulate>
__device__ __forceinline__ void umma_ss(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t lead) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 ad, bd;\n\tmov.b64 ad, {%1, %5};\n\tmov.b64 bd, {%2, %5};\n\t"
        "setp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %6, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], ad, bd, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(kIdesc), "n"(kAccumulate ? 1 : 0), "r"(kDescHi), "r"(lead)
        : "memory");
}
// A from tensor memory: lane = row, one 32-bit column = two consecutive k
template <uint32_t kIdesc>
__device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t accumulate, uint32_t lead) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 bd;\n\tmov.b64 bd, {%2, %5};\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %6, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], bd, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(kIdesc), "r"(accumulate), "r"(kDescHi), "r"(lead)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t *bar, uint32_t lead) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
        ::"r"(smem_u32(bar)), "r"(lead)
        : "memory");
}
// 1 in one lane of the (converged) warp
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t pred;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(pred));
    return pred;
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// the three-input maximum of sm_100
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// 32 consecutive f32 columns of this thread's TMEM lane, without the wait
__device__ __forceinline__ void tmem_ld32_nowait(uint32_t taddr, uint32_t *r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

// ---- q and k rows: half a warp per 128-element row, lane hl of it owning dims 8 hl .. 8 hl + 7 -----------------------------------
// Loading, rotating and storing are separate, so that a warp has several rows of loads in flight; everything is kept small,
// because a CTA runs this code once, out of a cold instruction cache (a version with a quarter of a row per lane and eight rows
// unrolled took 8 us for 57 tokens).
struct Row8 {
    uint4 r[2];    // raw activations: eight f32, or eight f16 in r[0]
    float4 a[4];   // (cos, sin) pairs: CHATGLM2 two float4 (four pairs), CHATGLM four (eight)
};
// Row s of a tensor whose head starts at element e_head.  s >= n_tok: zeros.  vec: rows are 16-byte (f32) or 8-byte (f16) aligned.
__device__ __forceinline__ void load_row8(Row8 &x, const PrefillSeq &ps, int rope_type, const float *base, long long e_head, long long stride,
                                          int s, int hl) {
    const SeqDev &sq = ps.sq;
    const bool f16 = (sq.flags & CGLM_SEQ_QKV_F16) != 0;
    x.r[0] = x.r[1] = make_uint4(0u, 0u, 0u, 0u);
    const long long e = e_head + s * stride + 8 * hl;
    if (s < sq.qlen) {
        if (ps.vec && f16) {
            const uint2 *p = reinterpret_cast<const uint2 *>(reinterpret_cast<const __half *>(base) + e);
            const uint2 u = __ldg(p), v = __ldg(p + 1);
            x.r[0] = make_uint4(u.x, u.y, v.x, v.y);
        } else if (ps.vec) {
            const uint4 *p = reinterpret_cast<const uint4 *>(base + e);
            x.r[0] = __ldg(p);
            x.r[1] = __ldg(p + 1);
        } else if (f16) {
            const unsigned short *p = reinterpret_cast<const unsigned short *>(base) + e;
            x.r[0] = make_uint4(p[0] | p[1] << 16, p[2] | p[3] << 16, p[4] | p[5] << 16, p[6] | p[7] << 16);
        } else {
            const uint32_t *p = reinterpret_cast<const uint32_t *>(base) + e;
            x.r[0] = make_uint4(p[0], p[1], p[2], p[3]);
            x.r[1] = make_uint4(p[4], p[5], p[6], p[7]);
        }
    }
    // Angles: by_position: the arena's table, indexed by the derived ids (chatglm.cpp:1142-1153, 1319-1327); otherwise the table
    // rope_table_kernel filled for this call, [stream][token].
    const int sc = min(s, sq.qlen - 1);
    if (rope_type == CGLM_ROPE_CHATGLM2) {           // dims [0, 64) as adjacent pairs: lanes 0..7, ladder steps 4 hl .. 4 hl + 3
        const float4 *t = reinterpret_cast<const float4 *>(ps.angles + static_cast<long long>(sc) * 32 + 4 * (hl & 7));
        x.a[0] = __ldg(t);
        x.a[1] = __ldg(t + 1);
    } else if (rope_type == CGLM_ROPE_CHATGLM) {     // each 64-dim half as pairs (i, i + 32): ladder steps 8 (hl & 3) .. + 7
        const bool second = hl >= 8;                 // by the position id, the second half by the block position id
        const int lim = sq.n_ctx - 2;
        const int row = ps.by_position ? (second ? max(sc - lim, 0) : min(sc, lim)) : (second ? sq.qlen + sc : sc);
        const float4 *t = reinterpret_cast<const float4 *>(ps.angles + static_cast<long long>(row) * 32 + 8 * (hl & 3));
#pragma unroll
        for (int i = 0; i < 4; ++i) x.a[i] = __ldg(t + i);
    }
}
// The rotated row.  Every product and sum rounded separately, in the order of rope_rotate().
__device__ __forceinline__ void rotate_row8(const Row8 &x, bool f16, int rope_type, int hl, float (&y)[8]) {
    const uint32_t w[8] = {x.r[0].x, x.r[0].y, x.r[0].z, x.r[0].w, x.r[1].x, x.r[1].y, x.r[1].z, x.r[1].w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 h = __half22float2(*reinterpret_cast<const __half2 *>(&w[i]));
        y[2 * i] = h.x;
        y[2 * i + 1] = h.y;
    }
    if (!f16) {
#pragma unroll
        for (int i = 0; i < 8; ++i) y[i] = __uint_as_float(w[i]);
    }
    if (rope_type == CGLM_ROPE_CHATGLM2) {
        const float4 a[2] = {x.a[0], x.a[1]};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float c = i & 1 ? a[i >> 1].z : a[i >> 1].x, s = i & 1 ? a[i >> 1].w : a[i >> 1].y;
            float y0, y1;
            rope_rotate(y[2 * i], y[2 * i + 1], c, s, y0, y1);
            if (hl < 8) { y[2 * i] = y0; y[2 * i + 1] = y1; }
        }
    } else if (rope_type == CGLM_ROPE_CHATGLM) {
        const bool upper = (hl & 4) != 0;   // holds x_{i + 32}; the pair's other element sits four lanes away
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float c = i & 1 ? x.a[i >> 1].z : x.a[i >> 1].x, s = i & 1 ? x.a[i >> 1].w : x.a[i >> 1].y;
            const float o = __shfl_xor_sync(0xffffffffu, y[i], 4);
            const float p = __fmul_rn(o, s), q = __fmul_rn(y[i], c);
            y[i] = upper ? __fadd_rn(p, q) : __fsub_rn(q, p);   // x_i: x c - o s; x_{i + 32}: o s + x c
        }
    }
}
__device__ __forceinline__ uint4 pack_half8(const float (&y)[8]) {
    return make_uint4(pack_half2(y[0], y[1]), pack_half2(y[2], y[3]), pack_half2(y[4], y[5]), pack_half2(y[6], y[7]));
}
__device__ __forceinline__ void st_f32x8(float *p, const float (&y)[8]) {
    if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {
        reinterpret_cast<float4 *>(p)[0] = make_float4(y[0], y[1], y[2], y[3]);
        reinterpret_cast<float4 *>(p)[1] = make_float4(y[4], y[5], y[6], y[7]);
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) p[i] = y[i];
    }
}

// table: f32 [stream][token][32 ladder steps][cos, sin]: only for explicit position ids, or an arena without a table
__global__ void __launch_bounds__(256)
rope_table_kernel(AttnShape sh, SeqDev sq, float2 *__restrict__ table) {
    const int S = sq.qlen;
    const int n_streams = sh.rope_type == CGLM_ROPE_CHATGLM ? 2 : 1;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_streams * S * 32) return;
    const int li = i & 31, t = (i >> 5) % S, st = (i >> 5) / S;
    int pos, block;
    derive_positions(sq, sh.rope_type, t, pos, block);
    float c, s;
    rope_cos_sin(st ? block : pos, li, sh.theta_scale, c, s);
    table[i] = make_float2(c, s);
}

// ---- launch 1: RoPE on k, append of K rows and V^T columns -----------------------------------------------------------------
// Grid: (64-token blocks of all sequences, kv heads, {K, V}).
//   K CTAs  half a warp per token row, eight rows of loads in flight per warp;
//   V CTAs  transpose [64 tokens][128 dims] through shared memory, so that a V^T cache row is written as 128 contiguous
//           bytes (16 per thread when the append position is a multiple of 8 tokens).
// Bound by latency for two kv heads (a few MB), by HBM for the 32 of ChatGLM-6B.  The q rows do not pass through here (staging
// them as f16 took 99 of the 810 us of an 8192-token prompt): the attention kernel rotates them on their way to shared memory.
constexpr int kAppTokens = 64;
constexpr int kAppThreads = 256;

__global__ void __launch_bounds__(kAppThreads)
prefill_append_kernel(const __grid_constant__ PrefillTable tab, AttnShape sh, uint16_t *__restrict__ k_base, uint16_t *__restrict__ v_base) {
    // Launched as a programmatic dependent: nothing is read or written before the previous kernel of the stream has
    // completed.  The attention kernel that follows may take its place as soon as every CTA here has passed that wait: its q
    // rows are then final, and it waits for this grid before it reads the cache.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // V^T tile: dim d's 64 tokens as eight 16-byte chunks, chunk c at place c ^ (d / 4 & 7): no bank conflicts either way
    __shared__ uint4 tile[kD][kAppTokens / 8];
    int si = 0;
    while (si + 1 < tab.n_seq && static_cast<int>(blockIdx.x) >= tab.seqs[si + 1].block_begin) ++si;
    const PrefillSeq &ps = tab.seqs[si];
    const SeqDev &sq = ps.sq;
    const int G = sh.G, M = sh.M, g = blockIdx.y;
    const int t_begin = (static_cast<int>(blockIdx.x) - ps.block_begin) * kAppTokens;
    const int n_tok = min(kAppTokens, sq.qlen - t_begin);
    const bool in_f16 = (sq.flags & CGLM_SEQ_QKV_F16) != 0, vec = ps.vec != 0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long row = static_cast<long long>(sq.slot) * G + g;
    constexpr int kRows = kAppTokens / (kAppThreads / 32);   // token rows per warp
    if (blockIdx.z == 0) {
        const int hl = lane & 15;
        Row8 x[kRows / 2];
#pragma unroll
        for (int u = 0; u < kRows / 2; ++u)
            load_row8(x[u], ps, sh.rope_type, sq.k, g * sq.kv_head_stride, sq.kv_tok_stride, t_begin + warp * kRows + 2 * u + (lane >> 4), hl);
#pragma unroll
        for (int u = 0; u < kRows / 2; ++u) {
            const int s = t_begin + warp * kRows + 2 * u + (lane >> 4);
            float y[8];
            rotate_row8(x[u], in_f16, sh.rope_type, hl, y);
            if (s < sq.qlen) {
                *reinterpret_cast<uint4 *>(k_base + (row * M + sq.kv_before + s) * kD + 8 * hl) = pack_half8(y);
                if (sq.k_roped) st_f32x8(sq.k_roped + (static_cast<long long>(s) * G + g) * kD + 8 * hl, y);
            }
        }
        return;
    }
    float4 x[kRows];
#pragma unroll
    for (int u = 0; u < kRows; ++u) {
        const int t = warp * kRows + u;
        const long long e = (t_begin + t) * sq.kv_tok_stride + g * sq.kv_head_stride + 4 * lane;
        x[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < n_tok) {
            if (in_f16) {
                if (vec) {
                    const uint2 v = __ldg(reinterpret_cast<const uint2 *>(reinterpret_cast<const __half *>(sq.v) + e));
                    x[u].x = __uint_as_float(v.x);   // widened behind the loop: nothing here waits for a load
                    x[u].y = __uint_as_float(v.y);
                } else {
                    const unsigned short *p = reinterpret_cast<const unsigned short *>(sq.v) + e;
                    x[u].x = __uint_as_float(p[0] | p[1] << 16);
                    x[u].y = __uint_as_float(p[2] | p[3] << 16);
                }
            } else if (vec) {
                x[u] = __ldg(reinterpret_cast<const float4 *>(sq.v + e));
            } else {
                x[u] = make_float4(__ldg(sq.v + e), __ldg(sq.v + e + 1), __ldg(sq.v + e + 2), __ldg(sq.v + e + 3));
            }
        }
    }
    if (in_f16) {
#pragma unroll
        for (int u = 0; u < kRows; ++u) {
            const uint32_t w0 = __float_as_uint(x[u].x), w1 = __float_as_uint(x[u].y);
            const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&w0)), c = __half22float2(*reinterpret_cast<const __half2 *>(&w1));
            x[u] = make_float4(a.x, a.y, c.x, c.y);
        }
    }
    static_assert(kRows == 8, "a warp's token rows are one 16-byte chunk of every dim");
    const int place = warp ^ (lane & 7);
    tile[4 * lane][place] = make_uint4(pack_half2(x[0].x, x[1].x), pack_half2(x[2].x, x[3].x), pack_half2(x[4].x, x[5].x), pack_half2(x[6].x, x[7].x));
    tile[4 * lane + 1][place] = make_uint4(pack_half2(x[0].y, x[1].y), pack_half2(x[2].y, x[3].y), pack_half2(x[4].y, x[5].y), pack_half2(x[6].y, x[7].y));
    tile[4 * lane + 2][place] = make_uint4(pack_half2(x[0].z, x[1].z), pack_half2(x[2].z, x[3].z), pack_half2(x[4].z, x[5].z), pack_half2(x[6].z, x[7].z));
    tile[4 * lane + 3][place] = make_uint4(pack_half2(x[0].w, x[1].w), pack_half2(x[2].w, x[3].w), pack_half2(x[4].w, x[5].w), pack_half2(x[6].w, x[7].w));
    __syncthreads();
    uint16_t *vrow0 = v_base + row * kD * M + sq.kv_before + t_begin;
    const bool vec_row = ((sq.kv_before + t_begin) & 7) == 0;   // M is a multiple of 8: every row is then 16-byte aligned
    for (int idx = threadIdx.x; idx < kD * (kAppTokens / 8); idx += kAppThreads) {
        const int d = idx / (kAppTokens / 8), c = idx % (kAppTokens / 8), t = 8 * c;
        if (t >= n_tok) continue;
        const uint4 v = tile[d][c ^ (d >> 2 & 7)];
        uint16_t *dst = vrow0 + static_cast<long long>(d) * M + t;
        if (vec_row && t + 8 <= n_tok) {
            *reinterpret_cast<uint4 *>(dst) = v;
        } else {
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                if (t + e < n_tok) dst[e] = static_cast<uint16_t>(e & 1 ? w[e >> 1] >> 16 : w[e >> 1] & 0xffffu);
            }
        }
    }
}

// ---- launch 2: attention ----------------------------------------------------------------------------------------------------
// What a CTA works on at a time: two q tiles (one in kPrefillSingle) that read the same kv head.
struct Unit {
    int seq;
    int g;            // kv head
    int head[2];      // q head of each group's tile
    int tile[2];      // q row tile of each group's tile
    int n_step;       // 64-token steps, the same for both groups (a tile that ends earlier sees masked steps)
    bool store1;      // false: there is no second tile, group 1 repeats the first one and stores nothing
};
__device__ __forceinline__ Unit unit_of(const PrefillTable &tab, const AttnShape &sh, int idx) {
    Unit un;
    un.seq = 0;
    while (un.seq + 1 < tab.n_seq && idx >= tab.seqs[un.seq + 1].unit_begin) ++un.seq;
    const PrefillSeq &ps = tab.seqs[un.seq];
    const int u = idx - ps.unit_begin, n_q = ps.n_q;
    un.store1 = true;
    // the longest row tiles first
    if (tab.mode == kPrefillSingle) {
        un.tile[0] = un.tile[1] = n_q - 1 - u / sh.H;
        un.head[0] = un.head[1] = u % sh.H;
    } else if (tab.mode == kPrefillPairHeads) {
        const int per_kv = (sh.R + 1) / 2, hu = u % (sh.G * per_kv);
        un.tile[0] = un.tile[1] = n_q - 1 - u / (sh.G * per_kv);
        un.head[0] = hu / per_kv * sh.R + 2 * (hu % per_kv);
        un.store1 = 2 * (hu % per_kv) + 1 < sh.R;
        un.head[1] = un.head[0] + (un.store1 ? 1 : 0);
    } else {
        const int p = (n_q + 1) / 2 - 1 - u / sh.H;
        un.tile[0] = 2 * p;
        un.store1 = 2 * p + 1 < n_q;
        un.tile[1] = un.tile[0] + (un.store1 ? 1 : 0);
        un.head[0] = un.head[1] = u % sh.H;
    }
    un.g = un.head[0] / sh.R;
    const int L = ps.sq.kv_before + ps.sq.qlen;
    const int end = sh.mask_type == CGLM_MASK_CAUSAL ? min(L, ps.sq.kv_before + (un.tile[1] + 1) * kQTile) : L;   // one past the last visible token
    un.n_step = (end + kStep - 1) / kStep;
    return un;
}
// The units are dealt to the CTAs in rows of gridDim.x, every other row backwards: the k-th unit of this CTA (past the end: none
// left).  Units come longest first, so the shares come out even.
__device__ __forceinline__ int unit_index(int k) {
    const int n = gridDim.x, b = blockIdx.x;
    return k * n + ((k & 1) ? n - 1 - b : b);
}

// q row pairs p0, p0 + step, ... of the unit's tiles (64 pairs per tile) by one warp: load, rotate, scale, round to f16 and
// store at the places of the swizzled A operand.  at(w): where tile w goes, shared memory or the global image of it; kRows row
// pairs have their loads in flight together.
template <int kPairs, class At>
__device__ __forceinline__ void stage_q(const PrefillSeq &ps, const AttnShape &sh, const Unit &un, int n_groups, int p0, int step, int lane, At at) {
    const SeqDev &sq = ps.sq;
    const int hl = lane & 15, sub = lane >> 4;
    const bool f16 = (sq.flags & CGLM_SEQ_QKV_F16) != 0;
#pragma unroll 1
    for (int p = p0; p < 64 * n_groups; p += kPairs * step) {
        Row8 x[kPairs];
#pragma unroll
        for (int u = 0; u < kPairs; ++u) {
            const int pu = min(p + u * step, 64 * n_groups - 1), w = pu >> 6, r = 2 * (pu & 63) + sub;   // past the end: the last pair again
            load_row8(x[u], ps, sh.rope_type, sq.q, (w ? un.head[1] : un.head[0]) * sq.q_head_stride, sq.q_tok_stride,
                      (w ? un.tile[1] : un.tile[0]) * kQTile + r, hl);
        }
#pragma unroll
        for (int u = 0; u < kPairs; ++u) {
            const int pu = min(p + u * step, 64 * n_groups - 1), w = pu >> 6, r = 2 * (pu & 63) + sub;
            float y[8];
            rotate_row8(x[u], f16, sh.rope_type, hl, y);
            const int s = (w ? un.tile[1] : un.tile[0]) * kQTile + r;
            if (sq.q_roped && s < sq.qlen) st_f32x8(sq.q_roped + (static_cast<long long>(s) * sh.H + (w ? un.head[1] : un.head[0])) * kD + 8 * hl, y);
#pragma unroll
            for (int i = 0; i < 8; ++i) y[i] = __fmul_rn(y[i], sh.scale);
            *reinterpret_cast<uint4 *>(at(w) + (hl >> 3) * kHalfBytes + r * 128 + (((hl & 7) ^ (r & 7)) << 4)) = pack_half8(y);
        }
    }
}
// 32 bytes of one thread to global memory: one full sector per lane
__device__ __forceinline__ void st_sector(void *p, const uint32_t (&v)[8], int align) {
    if (align >= 32) {
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]),
                     "r"(v[5]), "r"(v[6]), "r"(v[7])
                     : "memory");
    } else if (align >= 16) {
        reinterpret_cast<uint4 *>(p)[0] = make_uint4(v[0], v[1], v[2], v[3]);
        reinterpret_cast<uint4 *>(p)[1] = make_uint4(v[4], v[5], v[6], v[7]);
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) reinterpret_cast<uint2 *>(p)[i] = make_uint2(v[2 * i], v[2 * i + 1]);
    }
}

__global__ void __launch_bounds__(kThreads, 1)
prefill_attn_kernel(const __grid_constant__ CUtensorMap k_map, const __grid_constant__ PrefillTable tab, AttnShape sh, int n_units,
                    uint8_t *__restrict__ q_scratch, WsHeader *hdr) {
    extern __shared__ uint8_t smem_raw[];
    PrefillSmem &sm = *reinterpret_cast<PrefillSmem *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // the same in every lane, and known to be
    const int n_groups = tab.mode == kPrefillSingle ? 1 : 2;

    if (tid == 0) {
        sm.abort_flag = 0;
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&sm.kv_full[s], 1);
            mbar_init(&sm.kv_empty[s], n_groups);
        }
        for (int w = 0; w < 2; ++w) {
            mbar_init(&sm.q_full[w], 1);
            mbar_init(&sm.q_empty[w], 1);
            mbar_init(&sm.s_full[w], 1);
            mbar_init(&sm.s_empty[w], kGroupThreads / 32);
            mbar_init(&sm.p_full[w][0], kGroupThreads / 32);   // two: a group may be a step ahead of its MMA warp
            mbar_init(&sm.p_full[w][1], kGroupThreads / 32);
            mbar_init(&sm.o_step[w], 1);
            mbar_init(&sm.o_full[w], 1);
            mbar_init(&sm.o_empty[w], kGroupThreads / 32);
        }
        fence_mbar_init();
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, sm.tmem_base, 0);

    if (warp < kLoadWarp) {
        // The first unit's q rows straight into shared memory, by every warp that has nothing else to do yet.  They are the call's
        // input: final once the append kernel has started, which this grid's launch implies.
        const Unit un = unit_of(tab, sh, unit_index(0));   // the grid has no more CTAs than there are units
        stage_q<4>(tab.seqs[un.seq], sh, un, n_groups, warp, kLoadWarp, lane, [&](int w) { return sm.q[w]; });
        fence_proxy_async();   // plain stores above, the tensor core reads through the async proxy
        named_bar_sync(4, 32 * kLoadWarp);
        if (tid < n_groups) mbar_arrive(&sm.q_full[tid]);
        __syncwarp();
    }
    if (warp >= kQWarp) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegs));
        if (warp < kLoadWarp) {
            // ================================ q warps: tiles of the CTA's second and later units ===========================
            // The tile is staged in global memory (L2), already in the order of the swizzled operand, while the previous unit
            // runs, and copied in when that unit's last scores have been computed: a unit starts without a round trip for q.
            const int qw = warp - kQWarp;
            uint8_t *scratch = q_scratch + static_cast<size_t>(blockIdx.x) * 2 * kTileBytes;
            for (int k = 1, idx; (idx = unit_index(k)) < n_units; ++k) {
                const Unit un = unit_of(tab, sh, idx);
                const PrefillSeq &ps = tab.seqs[un.seq];
                if (k > 1) {   // the previous tiles have left the scratch
                    for (int w = 0; w < n_groups; ++w) mbar_wait_bounded(&sm.q_full[w], (k - 1) & 1, &sm.abort_flag);
                }
                __syncwarp();
                stage_q<2>(ps, sh, un, n_groups, qw, 4, lane, [&](int w) { return scratch + w * kTileBytes; });
                __threadfence();
                asm volatile("fence.proxy.async;" ::: "memory");   // plain stores above, the bulk copy reads through the async proxy
                named_bar_sync(3, 128);
                if (warp == kQWarp && lane == 0) {
                    asm volatile("fence.proxy.async;" ::: "memory");
                    for (int w = 0; w < n_groups; ++w) {
                        mbar_wait_bounded(&sm.q_empty[w], (k - 1) & 1, &sm.abort_flag);
                        mbar_arrive_expect_tx(&sm.q_full[w], kTileBytes);
                        bulk_load(sm.q[w], scratch + w * kTileBytes, kTileBytes, &sm.q_full[w]);
                    }
                }
                __syncwarp();
            }
        } else if (warp == kLoadWarp) {
            // ================================ load warp: K(0), V(0), K(1), V(1), ... through the ring =====================
            if (lane == 0) {
                tma_prefetch_desc(&k_map);
                asm volatile("griddepcontrol.wait;" ::: "memory");   // the append kernel's K rows and V^T columns are in place
                int st = 0;
                uint32_t parity = 1;   // a fresh barrier counts as the completed phase before its first one
                for (int k = 0, idx; (idx = unit_index(k)) < n_units; ++k) {
                    const Unit un = unit_of(tab, sh, idx);
                    const CUtensorMap *v_map = &tab.v_map[un.seq];
                    const int kv_row = tab.seqs[un.seq].sq.slot * sh.G + un.g, n_tiles = (un.n_step + 1) / 2;
                    for (int i = 0; i < 2 * n_tiles; ++i) {
                        const int j = i >> 1;
                        mbar_wait_bounded(&sm.kv_empty[st], parity, &sm.abort_flag);
                        mbar_arrive_expect_tx(&sm.kv_full[st], kTileBytes);
                        if ((i & 1) == 0) {
                            tma_load_3d(sm.kv[st], &k_map, 0, j * kKvTile, kv_row, &sm.kv_full[st]);
                            tma_load_3d(sm.kv[st] + kHalfBytes, &k_map, 64, j * kKvTile, kv_row, &sm.kv_full[st]);
                        } else {
                            tma_load_2d(sm.kv[st], v_map, j * kKvTile, kv_row * kD, &sm.kv_full[st]);
                            tma_load_2d(sm.kv[st] + kHalfBytes, v_map, j * kKvTile + 64, kv_row * kD, &sm.kv_full[st]);
                        }
                        if (++st == kStages) { st = 0; parity ^= 1; }
                    }
                }
                // every load of this CTA is on its way: the next kernel of the stream may take the places that free up
                asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
            }
        } else if (warp < kMmaWarp + n_groups) {
            // ================================ MMA warp of group w ========================================================
            // One warp per group: a wait of one leaves the tensor pipe to the other (one warp for both spent half of
            // its time between two MMAs).
            const int w = warp - kMmaWarp;
            const uint32_t kv_desc0 = desc_lo(smem_u32(sm.kv[0])), q_desc = desc_lo(smem_u32(sm.q[w]));
            const uint32_t t_s = tmem + 128 * w, t_o = tmem + 256 + 128 * w, lead = elect_one();
            // A place in the CTA's sequence of steps: step s (of n) of its k-th unit, the ring stage of its tile.  The scores
            // run one step ahead of the P V.
            struct Cursor {
                int k, s, n, st;
                uint32_t parity;
            };
            auto open = [&](Cursor &c) {   // first step of unit c.k, if there is one
                const int idx = unit_index(c.k);
                c.s = 0;
                c.n = idx < n_units ? unit_of(tab, sh, idx).n_step : 0;
            };
            auto advance = [&](Cursor &c) {
                ++c.s;
                if ((c.s & 1) == 0 || c.s == c.n) {   // K and V^T tiles alternate in the ring
                    c.st += 2;
                    if (c.st >= kStages) { c.st -= kStages; c.parity ^= 1; }
                }
                if (c.s == c.n) { ++c.k; open(c); }
            };
            Cursor cs{0, 0, 0, 0, 0}, cp{0, 0, 0, 1, 0};
            open(cs);
            open(cp);
            auto scores = [&](int t) {   // Q K^T of step cs, the CTA's t-th
                const int half = cs.s & 1;
                if (half == 0) mbar_wait_bounded(&sm.kv_full[cs.st], cs.parity, &sm.abort_flag);
                if (cs.s == 0) mbar_wait_bounded(&sm.q_full[w], cs.k & 1, &sm.abort_flag);
                if (t > 0) mbar_wait_bounded(&sm.s_empty[w], (t - 1) & 1, &sm.abort_flag);
                const uint32_t b = kv_desc0 + ((cs.st * kTileBytes + half * kStep * 128) >> 4);
                const bool last = cs.s + 1 == cs.n;
                __syncwarp();
                tc_fence_after();
                umma_ss<kIdescS, false>(t_s, q_desc, b, lead);
#pragma unroll
                for (int ks = 1; ks < 8; ++ks) {
                    const int off = ((ks >> 2) * kHalfBytes + (ks & 3) * 32) >> 4;
                    umma_ss<kIdescS, true>(t_s, q_desc + off, b + off, lead);
                }
                umma_commit(&sm.s_full[w], lead);
                if (half == 1 || last) umma_commit(&sm.kv_empty[cs.st], lead);
                if (last) umma_commit(&sm.q_empty[w], lead);
                advance(cs);
            };
            if (cs.n > 0) scores(0);
            for (int t = 0; cp.n > 0; ++t) {
                // the next scores as soon as the softmax has those of step t in registers; at the end of a unit, whose successor's q
                // tile may not be there yet, behind the P V
                const bool ahead = cs.n > 0 && cs.s > 0;
                if (ahead) scores(t + 1);
                const int half = cp.s & 1;
                if (half == 0) mbar_wait_bounded(&sm.kv_full[cp.st], cp.parity, &sm.abort_flag);
                if (cp.s == 0 && cp.k > 0) mbar_wait_bounded(&sm.o_empty[w], (cp.k - 1) & 1, &sm.abort_flag);
                mbar_wait_bounded(&sm.p_full[w][t & 1], (t >> 1) & 1, &sm.abort_flag);   // P(t) written, any rescale of O done
                const uint32_t b = kv_desc0 + ((cp.st * kTileBytes + half * kHalfBytes) >> 4);
                const uint32_t a = t_s + 64 + 32 * (t & 1);
                const bool last = cp.s + 1 == cp.n;
                __syncwarp();
                tc_fence_after();
                umma_ts<kIdescO>(t_o, a, b, cp.s != 0, lead);
#pragma unroll
                for (int ks = 1; ks < kStep / 16; ++ks) umma_ts<kIdescO>(t_o, a + 8 * ks, b + (ks * 32 >> 4), 1, lead);
                umma_commit(&sm.o_step[w], lead);
                if (half == 1 || last) umma_commit(&sm.kv_empty[cp.st], lead);
                if (last) umma_commit(&sm.o_full[w], lead);
                advance(cp);
                if (!ahead && cs.n > 0) scores(t + 1);
            }
        }
    } else {
        // ================================ softmax groups: one q row per thread ========================================
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSoftmaxRegs));
        const int w = warp >> 2, gw = warp & 3;   // group, warp inside it
        const int row = 32 * gw + lane;           // TMEM lane
        const uint32_t lane_base = static_cast<uint32_t>(32 * gw) << 16;   // this warp's quarter of the TMEM lanes
        const uint32_t ts = tmem + 128 * w + lane_base, to = tmem + 256 + 128 * w + lane_base;
        const bool causal = sh.mask_type == CGLM_MASK_CAUSAL;
        int t = 0;   // steps so far
        for (int k = 0, idx; w < n_groups && (idx = unit_index(k)) < n_units; ++k) {
            const Unit un = unit_of(tab, sh, idx);
            const PrefillSeq &ps = tab.seqs[un.seq];
            const SeqDev &sq = ps.sq;
            const int S = sq.qlen, h = w ? un.head[1] : un.head[0], s0 = (w ? un.tile[1] : un.tile[0]) * kQTile, n_step = un.n_step;
            float m_ref = kNoMax, l_run = 0.f;   // reference maximum (log2 domain) and row sum relative to it
            // the last token a row may attend (inclusive); a row past S is computed like any other and not stored
            const int L = sq.kv_before + S, s_row = s0 + row;
            const int row_last = causal ? min(L - 1, sq.kv_before + s_row) : (s_row < S - 1 ? L - 2 : L - 1);
            // One step: 64 tokens.  Masked and unmasked steps are separate code: in one loop the mask's selects are issued, if
            // predicated off, in every step.
            auto step = [&](int j, auto masked) {
                mbar_wait_bounded(&sm.s_full[w], t & 1, &sm.abort_flag);
                __syncwarp();   // aligned tensor-memory instructions follow
                tc_fence_after();
                float2 sv[kStep / 2];
                tmem_ld32_nowait(ts, reinterpret_cast<uint32_t *>(sv));
                tmem_ld32_nowait(ts + 32, reinterpret_cast<uint32_t *>(sv) + 32);
                tmem_wait_ld();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sm.s_empty[w]);   // the scores of the next step may follow
                // raw scores stay in sv; the log2(e) factor is folded into the exponent's FMA below.  Independent chains for
                // the maximum and the sum: one long dependent chain would cost more than the math.
                if constexpr (decltype(masked)::value) {
                    const int last = row_last - j * kStep;
#pragma unroll
                    for (int i = 0; i < kStep / 2; ++i) {
                        sv[i].x = 2 * i <= last ? sv[i].x : -INFINITY;
                        sv[i].y = 2 * i + 1 <= last ? sv[i].y : -INFINITY;
                    }
                }
                float mx4[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) mx4[c] = fmaxf(sv[c].x, sv[c].y);
#pragma unroll
                for (int i = 4; i < kStep / 2; ++i) mx4[i & 3] = max3(mx4[i & 3], sv[i].x, sv[i].y);
                const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * kLog2e;
                // keep the old reference unless the maximum outgrew it by more than the threshold
                const bool grow = mx > m_ref + kRescaleThreshold;   // also true for the first step with a score above -inf
                if (__any_sync(0xffffffffu, grow)) {
                    const float m_new = grow ? mx : m_ref;
                    const float alpha = grow ? ex2_approx(m_ref - m_new) : 1.f;   // 0 when m_ref was kNoMax
                    l_run *= alpha;
                    m_ref = m_new;
                    if (j > 0) {
                        // rescale this warp's rows of O: P V(t - 1) must have landed (P V(t - 2) has: it precedes the scores of t)
                        mbar_wait_bounded(&sm.o_step[w], (t - 1) & 1, &sm.abort_flag);
                        __syncwarp();
                        tc_fence_after();
#pragma unroll 1
                        for (int ch = 0; ch < 8; ++ch) {
                            uint32_t ov[16];
                            asm volatile(
                                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
                                "tcgen05.wait::ld.sync.aligned;"
                                : "=r"(ov[0]), "=r"(ov[1]), "=r"(ov[2]), "=r"(ov[3]), "=r"(ov[4]), "=r"(ov[5]), "=r"(ov[6]), "=r"(ov[7]),
                                  "=r"(ov[8]), "=r"(ov[9]), "=r"(ov[10]), "=r"(ov[11]), "=r"(ov[12]), "=r"(ov[13]), "=r"(ov[14]), "=r"(ov[15])
                                : "r"(to + ch * 16)
                                : "memory");
#pragma unroll
                            for (int i = 0; i < 16; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
                            tmem_st16(to + ch * 16, ov);
                        }
                    }
                }
                const float2 lg = make_float2(kLog2e, kLog2e), mb = make_float2(-m_ref, -m_ref);
                float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
                for (int ch = 0; ch < kStep / 32; ++ch) {
                    uint32_t packed[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        float2 e = __ffma2_rn(sv[16 * ch + i], lg, mb);   // masked scores are -inf: p = 0
                        e.x = ex2_approx(e.x);
                        e.y = ex2_approx(e.y);
                        sum[i & 1] = __fadd2_rn(sum[i & 1], e);
                        packed[i] = pack_half2(e.x, e.y);
                    }
                    // tokens [32 ch, 32 ch + 32) of the row: columns [16 ch, 16 ch + 16) of P.  The P V that read this buffer two
                    // steps ago precedes the scores of this step in the tensor pipe.
                    tmem_st16(ts + 64 + 32 * (t & 1) + ch * 16, packed);
                }
                l_run += (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sm.p_full[w][t & 1]);
                ++t;
            };
            // steps in which every row of this warp sees all 64 tokens
            const int first_last = causal ? min(L - 1, sq.kv_before + s0 + 32 * gw) : L - 2;
            const int n_clear = min(n_step, (first_last + 1) / kStep);
            int j = 0;
#pragma unroll 1
            for (; j < n_clear; ++j) step(j, std::false_type{});
#pragma unroll 1
            for (; j < n_step; ++j) step(j, std::true_type{});

            // ---- output: context_layer[s][h*D + d] (chatglm.cpp:712-717) straight from tensor memory, 32 bytes of its row per
            //      store and thread: whole sectors, nothing staged, nobody waited for ------------------------------------------
            mbar_wait_bounded(&sm.o_full[w], k & 1, &sm.abort_flag);
            __syncwarp();
            tc_fence_after();
            const float inv = 1.f / l_run;
            const bool out_f16 = (sq.flags & CGLM_SEQ_OUT_F16) != 0, store = s_row < S && (w == 0 || un.store1);
            const long long at = (static_cast<long long>(s_row) * sh.H + h) * kD;
            const int align = static_cast<int>(reinterpret_cast<uintptr_t>(sq.out) & 31) == 0 ? 32 : ((reinterpret_cast<uintptr_t>(sq.out) & 15) == 0 ? 16 : 8);
#pragma unroll
            for (int ch = 0; ch < 4; ++ch) {
                uint32_t r[32];
                tmem_ld32_nowait(to + ch * 32, r);
                tmem_wait_ld();
                if (ch == 3) {   // all of O has been read: the next unit's P V may overwrite it
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sm.o_empty[w]);
                }
                if (store) {
                    if (out_f16) {
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            uint32_t v[8];
#pragma unroll
                            for (int e = 0; e < 8; ++e)
                                v[e] = pack_half2(__uint_as_float(r[16 * c + 2 * e]) * inv, __uint_as_float(r[16 * c + 2 * e + 1]) * inv);
                            st_sector(reinterpret_cast<__half *>(sq.out) + at + 32 * ch + 16 * c, v, align);
                        }
                    } else {
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            uint32_t v[8];
#pragma unroll
                            for (int e = 0; e < 8; ++e) v[e] = __float_as_uint(__uint_as_float(r[8 * c + e]) * inv);
                            st_sector(sq.out + at + 32 * ch + 8 * c, v, align);
                        }
                    }
                }
                __syncwarp();
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
    if (sm.abort_flag && tid == 0) {
        atomicExch(&hdr->status, static_cast<int>(CGLM_ERR_TIMEOUT));
    }
}

}  // namespace

// angle table of one call's sequence with explicit position ids (or an arena without a table): f32 [stream][token][32][2]
size_t prefill_angle_bytes(int S) { return static_cast<size_t>(2) * S * 32 * sizeof(float2); }

// tab: n_seq, seqs[].sq and v_map[] filled by the caller; k_map covers the whole arena.  own_angles: room for
// prefill_angle_bytes of every sequence.
cudaError_t launch_prefill(const LaunchCtx &cx, PrefillTable &tab, const CUtensorMap &k_map, float2 *own_angles) {
    static PerDeviceOnce configured;
    const int smem_bytes = static_cast<int>(sizeof(PrefillSmem)) + 1024;
    if (configured.needed(cx.device)) {
        cudaError_t e = require_current_device(cx.device);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(prefill_attn_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
        if (e != cudaSuccess) return e;
        configured.mark(cx.device);
    }
    const AttnShape &sh = cx.shape;
    int launched = 2, blocks = 0;
    long long tiles = 0;
    for (int i = 0; i < tab.n_seq; ++i) {
        PrefillSeq &ps = tab.seqs[i];
        const int S = ps.sq.qlen;
        ps.n_q = (S + kQTile - 1) / kQTile;
        ps.block_begin = blocks;
        blocks += (S + kAppTokens - 1) / kAppTokens;
        tiles += static_cast<long long>(ps.n_q) * sh.H;
        ps.vec = decode_rows_aligned(ps.sq.q, ps.sq.k, ps.sq.v, ps.sq.q_head_stride, ps.sq.kv_head_stride, nullptr, nullptr,
                                     (ps.sq.flags & CGLM_SEQ_QKV_F16) != 0) &&
                 ps.sq.q_tok_stride % 4 == 0 && ps.sq.kv_tok_stride % 4 == 0;
        // Angles: positions derived from the token index lie inside the arena's table (one row per cache position);
        // explicit position ids may not, so such a sequence gets a table of its own first.
        ps.angles = cx.rope_tab;
        ps.by_position = 1;
        if (sh.rope_type != CGLM_ROPE_DISABLED && (ps.sq.position_ids || !cx.rope_tab || S > cx.rope_tab_len)) {
            const int n_entries = (sh.rope_type == CGLM_ROPE_CHATGLM ? 2 : 1) * S * 32;
            rope_table_kernel<<<(n_entries + 255) / 256, 256, 0, cx.stream>>>(sh, ps.sq, own_angles);
            ps.angles = own_angles;
            ps.by_position = 0;
            own_angles += static_cast<size_t>(2) * S * 32;
            ++launched;
        }
    }
    // One tile per CTA while all tiles still run at once (a short prompt: more SMs, and nothing to overlap with); otherwise two.
    tab.mode = tiles <= cx.n_sm ? kPrefillSingle : (sh.R > 1 ? kPrefillPairHeads : kPrefillPairTiles);
    int units = 0;
    for (int i = 0; i < tab.n_seq; ++i) {
        PrefillSeq &ps = tab.seqs[i];
        ps.unit_begin = units;
        units += tab.mode == kPrefillSingle ? ps.n_q * sh.H : (tab.mode == kPrefillPairHeads ? ps.n_q * sh.G * ((sh.R + 1) / 2) : (ps.n_q + 1) / 2 * sh.H);
    }
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // see griddepcontrol.wait in both kernels
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks, sh.G, 2);
    cfg.blockDim = dim3(kAppThreads);
    cfg.stream = cx.stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, prefill_append_kernel, tab, sh, cx.k_base, cx.v_base);
    if (e != cudaSuccess) return e;
    cfg.gridDim = dim3(units < cx.n_sm ? units : (cx.n_sm < kPrefillMaxCtas ? cx.n_sm : kPrefillMaxCtas));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem_bytes;
    e = cudaLaunchKernelEx(&cfg, prefill_attn_kernel, k_map, tab, sh, units, cx.q_tiles, cx.hdr);
    g_launch_count += launched;
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace cglm

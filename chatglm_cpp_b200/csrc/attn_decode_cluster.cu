// Fused RoPE + f16 KV append + decode attention for head_dim 128, one thread-block cluster per (sequence, kv head) item
// (sm_100a): the small launches of chatglm.cpp:655-717 for one-token sequences.
//
// What bounds a small launch is not bytes: a 513-token item is 0.26 MB.  It is the chain of latencies from the dependency
// wait to the last store, and code that runs once per launch (about a microsecond per 5 KiB of it that misses the
// instruction cache).  The persistent kernel pays for its generality there: descriptors and spans, a q tile handed over by a
// helper warp, TMA and its barriers, and at the end partials that travel through L2 to whoever counts to the last one
// (measured on one 512-token sequence: 2.2 us from the wait to the q tile, 2.0 us of fold, 3.4 us of counting, 7.8 us of
// merge).  Here
//   - K and V^T go from global memory straight into the registers of the warp that multiplies them, sixteen bytes per lane
//     and request: 32 tokens are 16 + 16 requests, the first 32 leave before the q rows are read, and those of the next 32
//     tokens leave as soon as the product that used the registers has issued;
//   - the contraction indices of both products are permuted so that a lane's sixteen bytes are MMA fragments as they are
//     (any order of the summands will do, as long as both operands use it): no shared memory, no barrier in the loop;
//   - the partial results of an item meet in distributed shared memory: one cluster barrier, and every thread block finishes
//     its share of the 128 dims.  No counters, no scratch memory.
// The item's tokens are dealt out 32 at a time to the 4 * kCta warps of the cluster in turn.
#include "common.cuh"
#include "decode_rope.cuh"

namespace cglm {

namespace {

constexpr int kD = 128;
constexpr int kRows = 16;             // MMA M = q heads per kv head, zero padded
constexpr int kWarps = 4;
constexpr int kThreads = kWarps * 32;
constexpr int kChunk = 32;            // tokens a warp takes at a time
constexpr int kQStride = 136;         // halfs per q row (272 B): the eight-byte fragment reads of a half warp cover all banks
// Asked for instead of what ClusterSmem takes: thread blocks of one launch then spread over the SMs (two would not fit one),
// every kernel of the step runs with the same split of an SM's memory, without which they could not share SMs at all, and a
// thread block of the Linear kernels (kFmSplitSmem) still fits beside.
constexpr int kSmemBytes = kDecodeClusterSmem;
constexpr int kRoundsAhead = 4;       // rounds of the cluster asked for in L2 before the wait
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
// Running maximum before the first score above -inf (none seen, or keys that overflowed f16): ex2(-inf - this) is 0, not NaN.
constexpr float kNoMax = -1.0e30f;

template <int kCap>
struct ClusterTable {
    int n_seq;
    const unsigned int *gate[2];      // see DecodeTable::gate
    unsigned int gate_value[2];
    SeqDev seqs[kCap];
};

struct __align__(16) ClusterSmem {
    float part[kWarps][kRows * kD];   // the warps' results; [0] then holds the thread block's
    float stats[kWarps][2 * kRows];   // the warps' row maxima and row sums; [0] then the thread block's
    __half q[kRows][kQStride];
    __half newk[kD], newv[kD];
    SeqDev sq;
    int abort_flag;
};

__device__ __forceinline__ uint32_t peer_addr(const void *p, int rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ float ld_peer(uint32_t a) {
    float x;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(a) : "memory");
    return x;
}
__device__ __forceinline__ float2 ld_peer2(uint32_t a) {
    float2 x;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(x.x), "=f"(x.y) : "r"(a) : "memory");
    return x;
}
__device__ __forceinline__ uint4 ld_cache16(const uint16_t *p) { return __ldcg(reinterpret_cast<const uint4 *>(p)); }

// Token of a chunk behind column n (0..7) of n-block b (0..3) of the scores: lane (r, c) of the PV product holds V^T of
// tokens 8c .. 8c + 7, and its k-step j takes tokens 8c + 4j .. 8c + 4j + 3 in the places of score columns 2c, 2c + 1 of
// blocks 2j and 2j + 1.
__device__ __forceinline__ int chunk_token(int n, int b) { return (n >> 1) * 8 + 2 * b + (n & 1); }

// kCta: thread blocks per cluster.
template <int kCta, int kCap>
__global__ void __launch_bounds__(kThreads, 2)
decode_cluster_kernel(const __grid_constant__ ClusterTable<kCap> tab, AttnShape sh, uint16_t *__restrict__ k_base,
                      uint16_t *__restrict__ v_base, WsHeader *hdr, const float2 *__restrict__ rope_tab, int rope_tab_len) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    ClusterSmem &sm = *reinterpret_cast<ClusterSmem *>(smem_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r8 = lane >> 2, c = lane & 3;
    const int G = sh.G, R = sh.R, M = sh.M;
    const int rank = static_cast<int>(blockIdx.x) % kCta, item = static_cast<int>(blockIdx.x) / kCta;
    const int seq = item / G, g = item - seq * G;

    if (warp == 0) {
        reinterpret_cast<uint32_t *>(&sm.sq)[lane] = reinterpret_cast<const uint32_t *>(&tab.seqs[seq])[lane];
        if (lane == 0) sm.abort_flag = 0;
    }
    const bool gated = tab.gate[0] != nullptr || tab.gate[1] != nullptr;
    __syncthreads();
    const int flags = sm.sq.flags;
    const long long row = static_cast<long long>(sm.sq.slot) * G + g;
    const uint16_t *const kc = k_base + row * M * kD, *const vc = v_base + row * kD * M;
    const int tok_first = rank * (kWarps * kChunk), tok_step = kCta * kWarps * kChunk;

    // ---- ahead of the dependency wait: requests into L2 only (what they bring is what the loads below read, whoever
    // writes it meanwhile).  Positions on the device may move until the wait; here they only size the requests.
    {
        int np = sm.sq.n_past;
        if (flags & CGLM_SEQ_N_PAST_DEVICE) np = *reinterpret_cast<const volatile int *>(sm.sq.n_past_dev);
        const int kv = (flags & CGLM_SEQ_N_PAST_DEVICE) ? min(max(np, 0) + sh.V, M - 1) : sm.sq.kv_before;
        const int end = min(kv + 8, M) & ~7;
        for (int t0 = tok_first, left = kRoundsAhead; t0 < end && left > 0; t0 += tok_step, --left) {
            const int n_tok = min(kWarps * kChunk, end - t0);   // a multiple of 8, as M is
            prefetch_l2(kc + static_cast<long long>(t0) * kD + tid * n_tok, static_cast<uint32_t>(n_tok) * 2u);
            prefetch_l2(vc + static_cast<long long>(tid) * M + t0, static_cast<uint32_t>(n_tok) * 2u);
        }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");

    // ---- the first chunk's requests, clamped to the cache: the attended length need not be known yet ------------------
    int tok0 = tok_first + warp * kChunk;
    uint4 kf[4][4], vf[16];
    auto load_k = [&](int t0) {
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const uint16_t *p = kc + static_cast<long long>(min(t0 + chunk_token(r8, b), M - 1)) * kD + 8 * c;
#pragma unroll
            for (int j = 0; j < 4; ++j) kf[b][j] = ld_cache16(p + 32 * j);
        }
    };
    auto load_v = [&](int t0) {
        const uint16_t *p = vc + static_cast<long long>(r8) * M + min(t0 + 8 * c, M - 8);
#pragma unroll
        for (int nb = 0; nb < 16; ++nb) { vf[nb] = ld_cache16(p); p += 8 * static_cast<long long>(M); }
    };
    int L = M;   // until the position is known
    if (!(flags & CGLM_SEQ_N_PAST_DEVICE)) L = sm.sq.kv_before + ((flags & CGLM_SEQ_NO_APPEND) ? 0 : 1);
    if (tok0 < L) { load_k(tok0); load_v(tok0); }

    // ---- q (every thread block), the new k and v ---------------------------------------------------------------------------
    int n_past = sm.sq.n_past, kv_before = sm.sq.kv_before;
    if (flags & CGLM_SEQ_N_PAST_DEVICE) {
        n_past = *reinterpret_cast<const volatile int *>(sm.sq.n_past_dev);
        const int np_max = M - sh.V - 1;   // the appended token must fit the cache
        if (n_past < 0 || n_past > np_max) {
            n_past = n_past < 0 ? 0 : np_max;
            if (tid == 0) atomicExch(&hdr->status, static_cast<int>(CGLM_ERR_INVALID_ARG));
        }
        kv_before = sh.V + n_past;   // CGLM_SEQ_USE_KV_LOCAL is not combined with a device-side position
        L = kv_before + ((flags & CGLM_SEQ_NO_APPEND) ? 0 : 1);
    }
    const bool append = !(flags & CGLM_SEQ_NO_APPEND);
    if (gated) {   // host-buffer call: the activations are in place / the output is free once these words are written
        if (tid == 0) {
            for (int gi = 0; gi < 2; ++gi) {
                if (tab.gate[gi] && !wait_gate(tab.gate[gi], tab.gate_value[gi], &sm.abort_flag)) sm.abort_flag = 1;
            }
            if (sm.abort_flag) atomicExch(&hdr->status, static_cast<int>(CGLM_ERR_TIMEOUT));
        }
        __syncthreads();
    }
    {
        // warp w takes q rows 4w .. 4w + 3, warp 0 the new k and warp 1 the new v as well; lane l dims 4l .. 4l + 3
        const bool f16 = (flags & CGLM_SEQ_QKV_F16) != 0;
        const bool k_row = warp == 0 && (append || sm.sq.k_roped != nullptr), v_row = warp == 1 && append;
        auto ld4 = [&](const float *base, long long e) -> float4 {   // element index either way
            if (!f16) return __ldcg(reinterpret_cast<const float4 *>(base + e));
            const uint2 u = __ldcg(reinterpret_cast<const uint2 *>(reinterpret_cast<const __half *>(base) + e));
            const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&u.x)), b = __half22float2(*reinterpret_cast<const __half2 *>(&u.y));
            return make_float4(a.x, a.y, b.x, b.y);
        };
        float4 x[5], xv;
        x[4] = xv = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = 4 * warp + i;
            x[i] = r < R ? ld4(sm.sq.q, (static_cast<long long>(g) * R + r) * sm.sq.q_head_stride + 4 * lane) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (k_row) x[4] = ld4(sm.sq.k, g * sm.sq.kv_head_stride + 4 * lane);
        if (v_row) xv = ld4(sm.sq.v, g * sm.sq.kv_head_stride + 4 * lane);
        const int mode = (flags & CGLM_SEQ_Q_ROPED) ? static_cast<int>(CGLM_ROPE_DISABLED) : sh.rope_type;
        if (mode != CGLM_ROPE_DISABLED) {
            int pos_id = 0, block_id = 0;
            float2 cs0, cs1 = make_float2(1.f, 0.f);
            SeqDev ps = sm.sq;
            ps.n_past = n_past;
            derive_positions(ps, mode, 0, pos_id, block_id);
            cs0 = rope_angle(pos_id, lane, sh.theta_scale, rope_tab, rope_tab_len);
            if (mode == CGLM_ROPE_CHATGLM) cs1 = rope_angle(block_id, lane, sh.theta_scale, rope_tab, rope_tab_len);
            rope_rows<5>(x, mode, lane, cs0, cs1);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = 4 * warp + i;
            *reinterpret_cast<uint2 *>(&sm.q[r][4 * lane]) = pack_half4(__fmul_rn(x[i].x, sh.scale), __fmul_rn(x[i].y, sh.scale),
                                                                       __fmul_rn(x[i].z, sh.scale), __fmul_rn(x[i].w, sh.scale));
            if (rank == 0 && sm.sq.q_roped && r < R) {
                *reinterpret_cast<float4 *>(sm.sq.q_roped + (static_cast<long long>(g) * R + r) * kD + 4 * lane) = x[i];
            }
        }
        if (k_row) {
            if (rank == 0 && sm.sq.k_roped) *reinterpret_cast<float4 *>(sm.sq.k_roped + static_cast<long long>(g) * kD + 4 * lane) = x[4];
            if (append) {
                const uint2 h = pack_half4(x[4].x, x[4].y, x[4].z, x[4].w);
                *reinterpret_cast<uint2 *>(&sm.newk[4 * lane]) = h;
                if (rank == 0) *reinterpret_cast<uint2 *>(k_base + (row * M + kv_before) * kD + 4 * lane) = h;
            }
        }
        if (v_row) {
            const uint2 h = pack_half4(xv.x, xv.y, xv.z, xv.w);
            *reinterpret_cast<uint2 *>(&sm.newv[4 * lane]) = h;
            if (rank == 0) {
                uint16_t *col = v_base + (row * kD + 4 * lane) * M + kv_before;
                col[0] = static_cast<uint16_t>(h.x & 0xffffu);
                col[M] = static_cast<uint16_t>(h.x >> 16);
                col[2 * static_cast<long long>(M)] = static_cast<uint16_t>(h.y & 0xffffu);
                col[3 * static_cast<long long>(M)] = static_cast<uint16_t>(h.y >> 16);
            }
        }
    }
    __syncthreads();

    // ---- this warp's chunks ---------------------------------------------------------------------------------------------------
    float o[16][4];
#pragma unroll
    for (int i = 0; i < 16; ++i) { o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f; }
    float m_run[2] = {kNoMax, kNoMax}, l_run[2] = {0.f, 0.f};   // rows r8 and r8 + 8; this lane's share of the sums
    const __half *const qa = &sm.q[r8][8 * c], *const qb = &sm.q[r8 + 8][8 * c];
#pragma unroll 1
    for (; tok0 < L; tok0 += tok_step) {
        const bool last = tok0 + kChunk >= L;   // holds the item's last token: the appended one, then stale cache
        if (last && append) {
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                if (tok0 + chunk_token(r8, b) == kv_before) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) kf[b][j] = *reinterpret_cast<const uint4 *>(&sm.newk[32 * j + 8 * c]);
                }
            }
        }
        // scores: k-step (j, h) takes dims 32j + 8c + 4h .. + 3 of every lane c
        float s[4][4];
#pragma unroll
        for (int b = 0; b < 4; ++b) { s[b][0] = s[b][1] = s[b][2] = s[b][3] = 0.f; }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint4 qr = *reinterpret_cast<const uint4 *>(qa + 32 * j), qs = *reinterpret_cast<const uint4 *>(qb + 32 * j);
            const uint32_t a0[4] = {qr.x, qs.x, qr.y, qs.y}, a1[4] = {qr.z, qs.z, qr.w, qs.w};
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                mma_m16n8k16(s[b], a0, kf[b][j].x, kf[b][j].y);
                mma_m16n8k16(s[b], a1, kf[b][j].z, kf[b][j].w);
            }
        }
        if (tok0 + tok_step < L) load_k(tok0 + tok_step);
        // online softmax in the log2 domain
        float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int b = 0; b < 4; ++b) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                s[b][e] = tok0 + 8 * c + 2 * b + (e & 1) < L ? s[b][e] * kLog2e : -INFINITY;
                mx[e >> 1] = fmaxf(mx[e >> 1], s[b][e]);
            }
        }
        float alpha[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
            mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
            const float m_new = fmaxf(m_run[h], mx[h]);
            alpha[h] = ex2_approx(m_run[h] - m_new);
            m_run[h] = m_new;
            l_run[h] *= alpha[h];
        }
        uint32_t pa[2][4];   // A fragments of the two k-steps of PV
#pragma unroll
        for (int b = 0; b < 4; ++b) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float p0 = ex2_approx(s[b][2 * h] - m_run[h]), p1 = ex2_approx(s[b][2 * h + 1] - m_run[h]);
                l_run[h] += p0 + p1;
                pa[b >> 1][2 * (b & 1) + h] = pack_half2(p0, p1);
            }
        }
        if (last) {   // tokens past the attended length hold stale values (0 x NaN is NaN), the appended one is not in the cache yet
            const int keep_end = append ? kv_before : L;
            uint32_t keep[4], ins[4];
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                const int t = tok0 + 8 * c + 2 * w;
                keep[w] = (t < keep_end ? 0x0000ffffu : 0u) | (t + 1 < keep_end ? 0xffff0000u : 0u);
                ins[w] = !append ? 0u : (t == kv_before ? 0x0000ffffu : 0u) | (t + 1 == kv_before ? 0xffff0000u : 0u);
            }
#pragma unroll
            for (int nb = 0; nb < 16; ++nb) {
                const uint32_t nv = append ? __half_as_ushort(sm.newv[8 * nb + r8]) * 0x00010001u : 0u;
                vf[nb].x = (vf[nb].x & keep[0]) | (nv & ins[0]);
                vf[nb].y = (vf[nb].y & keep[1]) | (nv & ins[1]);
                vf[nb].z = (vf[nb].z & keep[2]) | (nv & ins[2]);
                vf[nb].w = (vf[nb].w & keep[3]) | (nv & ins[3]);
            }
        }
#pragma unroll
        for (int nb = 0; nb < 16; ++nb) {
            o[nb][0] *= alpha[0]; o[nb][1] *= alpha[0]; o[nb][2] *= alpha[1]; o[nb][3] *= alpha[1];
            mma_m16n8k16(o[nb], pa[0], vf[nb].x, vf[nb].y);
            mma_m16n8k16(o[nb], pa[1], vf[nb].z, vf[nb].w);
        }
        if (tok0 + tok_step < L) load_v(tok0 + tok_step);
    }
    // Nothing is left to load: the next kernel may come up and ask for what it can (earlier, its requests would stand in
    // front of this kernel's: 825 against 844 us per replay of a 28-layer step of one 512-token chat)
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    // ---- the four warps of the thread block ----------------------------------------------------------------------------------
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], 1);
        l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], 2);
        if (c == 0) {
            sm.stats[warp][r8 + 8 * h] = m_run[h];
            sm.stats[warp][kRows + r8 + 8 * h] = l_run[h];
        }
    }
    __syncthreads();
    {
        float a[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = r8 + 8 * h;
            const float m_star = fmaxf(fmaxf(sm.stats[0][r], sm.stats[1][r]), fmaxf(sm.stats[2][r], sm.stats[3][r]));
            a[h] = ex2_approx(m_run[h] - m_star);
        }
        // float2 unit u of row r lives at unit u ^ 4(r & 3): conflict-free stores here, and 16-byte reads below
        float *mine = sm.part[warp];
        const int swz = 4 * (r8 & 3);
#pragma unroll
        for (int nb = 0; nb < 16; ++nb) {
            const int u = (4 * nb + c) ^ swz;
            *reinterpret_cast<float2 *>(&mine[r8 * kD + 2 * u]) = make_float2(o[nb][0] * a[0], o[nb][1] * a[0]);
            *reinterpret_cast<float2 *>(&mine[(r8 + 8) * kD + 2 * u]) = make_float2(o[nb][2] * a[1], o[nb][3] * a[1]);
        }
    }
    float m_cta = 0.f, l_cta = 0.f;   // of row tid, threads 0..15
    if (tid < kRows) {
        m_cta = fmaxf(fmaxf(sm.stats[0][tid], sm.stats[1][tid]), fmaxf(sm.stats[2][tid], sm.stats[3][tid]));
#pragma unroll
        for (int w = 0; w < kWarps; ++w) l_cta += sm.stats[w][kRows + tid] * ex2_approx(sm.stats[w][tid] - m_cta);
    }
    __syncthreads();
    if (tid < kRows) {
        sm.stats[0][tid] = m_cta;
        sm.stats[0][kRows + tid] = l_cta;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {   // each thread the same four float4 of all four copies
        float4 *p = reinterpret_cast<float4 *>(sm.part[0]) + i * kThreads + tid;
        const float4 v0 = p[0], v1 = p[kRows * kD / 4], v2 = p[2 * (kRows * kD / 4)], v3 = p[3 * (kRows * kD / 4)];
        p[0] = make_float4(((v0.x + v1.x) + v2.x) + v3.x, ((v0.y + v1.y) + v2.y) + v3.y, ((v0.z + v1.z) + v2.z) + v3.z,
                           ((v0.w + v1.w) + v2.w) + v3.w);
    }
    cluster_sync();

    // ---- the thread blocks of the cluster: rank k finishes dims [128 k / kCta, 128 (k + 1) / kCta) of the rows -------------
    // Only values that reach a store below are read from the peers: what keeps a peer's shared memory alive past these reads is
    // that the stores, and so the values, come before this thread's last arrival.
    if ((tid >> 3) < R && L > 0 && !sm.abort_flag) {
        constexpr int kUnits = kRows / kCta / 2 > 0 ? kRows / kCta / 2 : 1;   // float2 units per thread, eight threads per row
        const int r = tid >> 3, u0 = rank * (kD / 2 / kCta) + (tid & 7) * kUnits;
        const float *stat = &sm.stats[0][r];
        const bool want_l = !(flags & CGLM_SEQ_PARTIAL) || (rank == 0 && (tid & 7) == 0);
        float m[kCta], l[kCta];
        float2 v[kCta][kUnits];
#pragma unroll
        for (int k = 0; k < kCta; ++k) {
            m[k] = ld_peer(peer_addr(stat, k));
            l[k] = want_l ? ld_peer(peer_addr(stat + kRows, k)) : 0.f;
#pragma unroll
            for (int i = 0; i < kUnits; ++i) v[k][i] = ld_peer2(peer_addr(&sm.part[0][r * kD + 2 * ((u0 + i) ^ (4 * (r & 3)))], k));
        }
        float m_star = kNoMax, den = 0.f;
        float2 acc[kUnits];
#pragma unroll
        for (int k = 0; k < kCta; ++k) m_star = fmaxf(m_star, m[k]);
#pragma unroll
        for (int i = 0; i < kUnits; ++i) acc[i] = make_float2(0.f, 0.f);
#pragma unroll
        for (int k = 0; k < kCta; ++k) {
            const float w = ex2_approx(m[k] - m_star);
            den += w * l[k];
#pragma unroll
            for (int i = 0; i < kUnits; ++i) { acc[i].x += w * v[k][i].x; acc[i].y += w * v[k][i].y; }
        }
        const int head = g * R + r;
        if (flags & CGLM_SEQ_PARTIAL) {
            float *po = sm.sq.partial + static_cast<long long>(head) * (kD + 2);
#pragma unroll
            for (int i = 0; i < kUnits; ++i) *reinterpret_cast<float2 *>(po + 2 * (u0 + i)) = acc[i];
            if (rank == 0 && (tid & 7) == 0) { po[kD] = m_star * kLn2; po[kD + 1] = den; }
        } else {
            const float inv = 1.f / den;
#pragma unroll
            for (int i = 0; i < kUnits; ++i) {
                const long long e = static_cast<long long>(head) * kD + 2 * (u0 + i);
                if (flags & CGLM_SEQ_OUT_F16) {
                    *reinterpret_cast<uint32_t *>(reinterpret_cast<__half *>(sm.sq.out) + e) = pack_half2(acc[i].x * inv, acc[i].y * inv);
                } else {
                    *reinterpret_cast<float2 *>(sm.sq.out + e) = make_float2(acc[i].x * inv, acc[i].y * inv);
                }
            }
        }
    }
    // Nothing to order, and the output stores are not waited for.
    __syncwarp();
    asm volatile("barrier.cluster.arrive.relaxed.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

template <int kCta, int kCap>
cudaError_t configure(int device) {
    static PerDeviceOnce configured;
    if (!configured.needed(device)) return cudaSuccess;
    cudaError_t e = require_current_device(device);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(decode_cluster_kernel<kCta, kCap>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e == cudaSuccess) configured.mark(device);
    return e;
}

template <int kCta, int kCap>
cudaError_t launch(const LaunchCtx &cx, const DecodeTable &tab) {
    static thread_local ClusterTable<kCap> t;
    cudaError_t e = configure<kCta, kCap>(cx.device);
    if (e != cudaSuccess) return e;
    t.n_seq = tab.n_seq;
    for (int i = 0; i < 2; ++i) { t.gate[i] = tab.gate[i]; t.gate_value[i] = tab.gate_value[i]; }
    for (int i = 0; i < tab.n_seq; ++i) t.seqs[i] = tab.seqs[i];
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = kCta; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(tab.n_seq * cx.shape.G * kCta));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.stream = cx.stream;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    e = cudaLaunchKernelEx(&cfg, decode_cluster_kernel<kCta, kCap>, t, cx.shape, cx.k_base, cx.v_base, cx.hdr, cx.rope_tab,
                                       cx.rope_tab_len);
    g_launch_count += 1;
    return e != cudaSuccess ? e : cudaGetLastError();
}

template <int kCta>
int resident(int device) {
    static std::atomic<int> known[kMaxDevices];   // 1 + the count, 0: not asked yet
    const bool keep = device >= 0 && device < kMaxDevices;
    const int k = keep ? known[device].load(std::memory_order_relaxed) : 0;
    if (k > 0) return k - 1;
    if (configure<kCta, 8>(device) != cudaSuccess) return 0;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kCta; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kCta);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, decode_cluster_kernel<kCta, 8>, &cfg) != cudaSuccess) return 0;
    if (keep) known[device].store(n + 1, std::memory_order_relaxed);
    return n;
}

}  // namespace

int decode_cluster_resident(int device, int n_cta) {
    return n_cta == 8 ? resident<8>(device) : (n_cta == 4 ? resident<4>(device) : resident<2>(device));
}

cudaError_t launch_decode_cluster(const LaunchCtx &cx, const DecodeTable &tab, int n_cta) {
    static_assert(kDecodeClusterMaxSeq == 64, "the larger table");
    if (tab.n_seq <= 8) {
        switch (n_cta) {
        case 8: return launch<8, 8>(cx, tab);
        case 4: return launch<4, 8>(cx, tab);
        default: return launch<2, 8>(cx, tab);
        }
    }
    switch (n_cta) {
    case 8: return launch<8, 64>(cx, tab);
    case 4: return launch<4, 64>(cx, tab);
    default: return launch<2, 64>(cx, tab);
    }
}

}  // namespace cglm

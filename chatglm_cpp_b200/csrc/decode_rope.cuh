// What the decode kernels share: the rotation of head rows held four dims per lane, angles, requests into L2, the wait for
// a copy engine's word.
#pragma once
#include "common.cuh"

namespace cglm {
namespace {

__device__ __forceinline__ float4 ldg4(const float *p) { return __ldg(reinterpret_cast<const float4 *>(p)); }
__device__ __forceinline__ uint2 pack_half4(float a, float b, float c, float d) {
    return make_uint2(pack_half2(a, b), pack_half2(c, d));
}
// Angle of a position the arena's table does not hold (explicit position ids beyond the cache capacity): out of
// line, so that the double-precision sincos stays out of the instruction stream of the common case.
__device__ __noinline__ float2 rope_angle_uncached(int pos, int i, float theta_scale) {
    float2 cs;
    rope_cos_sin(pos, i, theta_scale, cs.x, cs.y);
    return cs;
}

__device__ __forceinline__ float2 rope_angle(int pos, int i, float theta_scale, const float2 *__restrict__ rope_tab, int rope_tab_len) {
    return pos >= 0 && pos < rope_tab_len ? __ldg(rope_tab + static_cast<long long>(pos) * 32 + i) : rope_angle_uncached(pos, i, theta_scale);
}

// Rotation of kN head rows in place: lane l holds dims 4l .. 4l + 3 of each, and ladder angle l of the position stream in
// cs0 (in CGLM_ROPE_CHATGLM mode that of the block-position stream in cs1).  Every product and sum is rounded separately and in the order of
// rope_rotate(): y0 = x0 c - x1 s, y1 = x0 s + x1 c.
template <int kN>
__device__ __forceinline__ void rope_rows(float4 (&x)[kN], int mode, int lane, float2 cs0, float2 cs1) {
    if (mode == CGLM_ROPE_CHATGLM2) {
        // lanes 0..15 hold pairs 2l and 2l+1 entirely; lanes 16..31 hold dims that do not rotate
        const int a = (2 * lane) & 31;
        const float ca = __shfl_sync(0xffffffffu, cs0.x, a), sa = __shfl_sync(0xffffffffu, cs0.y, a);
        const float cb = __shfl_sync(0xffffffffu, cs0.x, a + 1), sb = __shfl_sync(0xffffffffu, cs0.y, a + 1);
        const bool rot = lane < 16;
#pragma unroll
        for (int r = 0; r < kN; ++r) {
            float4 y;
            rope_rotate(x[r].x, x[r].y, ca, sa, y.x, y.y);
            rope_rotate(x[r].z, x[r].w, cb, sb, y.z, y.w);
            if (rot) x[r] = y;
        }
    } else if (mode == CGLM_ROPE_CHATGLM) {
        // lane l holds x_i (bit 3 of l clear) or x_{i+32} (set) of four pairs; the other element sits in lane l ^ 8
        const bool second = lane >= 16, upper = (lane & 8) != 0;
        float c[4], sg[4];   // sg: the sine with the sign this lane's element takes (-s for x_i, +s for x_{i+32})
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int a = 4 * (lane & 7) + e;
            const float c0 = __shfl_sync(0xffffffffu, cs0.x, a), s0 = __shfl_sync(0xffffffffu, cs0.y, a);
            const float c1 = __shfl_sync(0xffffffffu, cs1.x, a), s1 = __shfl_sync(0xffffffffu, cs1.y, a);
            c[e] = second ? c1 : c0;
            sg[e] = second ? s1 : s0;
        }
#pragma unroll
        for (int r = 0; r < kN; ++r) {
            const float ox = __shfl_xor_sync(0xffffffffu, x[r].x, 8), oy = __shfl_xor_sync(0xffffffffu, x[r].y, 8);
            const float oz = __shfl_xor_sync(0xffffffffu, x[r].z, 8), ow = __shfl_xor_sync(0xffffffffu, x[r].w, 8);
            // x_i:      y = x c - o s  (rope_rotate's y0 with x0 = x, x1 = o)
            // x_{i+32}: y = o s + x c  (rope_rotate's y1 with x0 = o, x1 = x); the sum commutes exactly
            const float px = __fmul_rn(ox, sg[0]), py = __fmul_rn(oy, sg[1]), pz = __fmul_rn(oz, sg[2]), pw = __fmul_rn(ow, sg[3]);
            x[r].x = upper ? __fadd_rn(px, __fmul_rn(x[r].x, c[0])) : __fsub_rn(__fmul_rn(x[r].x, c[0]), px);
            x[r].y = upper ? __fadd_rn(py, __fmul_rn(x[r].y, c[1])) : __fsub_rn(__fmul_rn(x[r].y, c[1]), py);
            x[r].z = upper ? __fadd_rn(pz, __fmul_rn(x[r].z, c[2])) : __fsub_rn(__fmul_rn(x[r].z, c[2]), pz);
            x[r].w = upper ? __fadd_rn(pw, __fmul_rn(x[r].w, c[3])) : __fsub_rn(__fmul_rn(x[r].w, c[3]), pw);
        }
    }
}

__device__ __forceinline__ void prefetch_l2(const void *p, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
// Polls a word that a copy engine writes, with a bound; false when it ran out.
__device__ __forceinline__ bool wait_gate(const unsigned int *word, unsigned int value, volatile int *abort_flag) {
    unsigned long long t0 = 0, now;
    for (unsigned int spin = 0; spin < kSpinLimit && !*abort_flag; ++spin) {
        unsigned int v;
        asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(word) : "memory");
        if (v == value) return true;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        if (t0 == 0) t0 = now;
        if (now - t0 > kGateLimitNs) break;
        __nanosleep(200);
    }
    return false;
}

}  // namespace
}  // namespace cglm

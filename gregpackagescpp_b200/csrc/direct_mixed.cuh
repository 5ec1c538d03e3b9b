// Building blocks of the mixed-precision direct-sum kernels.
#pragma once

#include "gtd_internal.cuh"

namespace gtd {

__device__ __forceinline__ float rsqrt_approx(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ void kahan_add(double &sum, double &comp, double v) {
    const double y = v - comp;
    const double t = sum + y;
    comp = (t - sum) - y;
    sum = t;
}

// FP64 Kahan accumulators of the I i-bodies of a thread: in registers, or (SMEM) in shared memory,
// which they only touch once per fold; the latter frees 12 registers per i-body for occupancy.
template <int I, bool SMEM, int T = kThreads>
struct KahanAcc;

template <int I, int T>
struct KahanAcc<I, false, T> {
    double s[3][I], c[3][I];
    __device__ __forceinline__ void init(int) {
#pragma unroll
        for (int d = 0; d < 3; ++d)
#pragma unroll
            for (int k = 0; k < I; ++k) s[d][k] = c[d][k] = 0.0;
    }
    __device__ __forceinline__ void add(int d, int k, double v) { kahan_add(s[d][k], c[d][k], v); }
    __device__ __forceinline__ double result(int d, int k) const { return s[d][k] - c[d][k]; }
};

template <int I, int T>
struct KahanAcc<I, true, T> {
    double (*sm)[I][T];  // [6][I][T]: sums x y z, compensations x y z
    int t;
    __device__ __forceinline__ void init(int tid) {
        t = tid;
#pragma unroll
        for (int d = 0; d < 6; ++d)
#pragma unroll
            for (int k = 0; k < I; ++k) sm[d][k][t] = 0.0;
    }
    __device__ __forceinline__ void add(int d, int k, double v) {
        double s = sm[d][k][t], c = sm[3 + d][k][t];
        kahan_add(s, c, v);
        sm[d][k][t] = s;
        sm[3 + d][k][t] = c;
    }
    __device__ __forceinline__ double result(int d, int k) const { return sm[d][k][t] - sm[3 + d][k][t]; }
};

// Order-preserving map of a float onto an unsigned int, so that warp minima and maxima of floats
// are single REDUX operations (__reduce_min_sync / __reduce_max_sync).
__device__ __forceinline__ unsigned f2key(float f) {
    const unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key2f(unsigned k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}
__device__ __forceinline__ float warp_minf(float v) { return key2f(__reduce_min_sync(0xffffffffu, f2key(v))); }
__device__ __forceinline__ float warp_maxf(float v) { return key2f(__reduce_max_sync(0xffffffffu, f2key(v))); }

// One staged body: FP32 hi part of x - c, its FP32 remainder lo, and G m.  Padding bodies are far
// away and massless, so their terms are exactly 0 on both paths.
__device__ __forceinline__ void stage_body(bool have, const double4 &q, const double3 &c, double G, int slot,
                                           float *hx, float *hy, float *hz, float *hm, float *lx, float *ly,
                                           float *lz) {
    if (have) {
        const double ex = q.x - c.x, ey = q.y - c.y, ez = q.z - c.z;
        const float fx = (float)ex, fy = (float)ey, fz = (float)ez;
        hx[slot] = fx;
        hy[slot] = fy;
        hz[slot] = fz;
        lx[slot] = (float)(ex - (double)fx);
        ly[slot] = (float)(ey - (double)fy);
        lz[slot] = (float)(ez - (double)fz);
        hm[slot] = (float)(G * q.w);
    } else {
        const float kFar = 1e30f;
        hx[slot] = hy[slot] = hz[slot] = kFar;
        lx[slot] = ly[slot] = lz[slot] = 0.f;
        hm[slot] = 0.f;
    }
}

// Bounding box of the 32 bodies a warp just staged (padding bodies left out), written by lane 0 to
// box[warp][6] of the buffer.  Every lane of the warp calls it.
__device__ __forceinline__ void stage_box(bool have, const float *hx, const float *hy, const float *hz, int slot,
                                          float *box) {
    const float kInf = __int_as_float(0x7f800000);
    const float x = hx[slot], y = hy[slot], z = hz[slot];
    const float lx = warp_minf(have ? x : kInf), ly = warp_minf(have ? y : kInf), lz = warp_minf(have ? z : kInf);
    const float ux = warp_maxf(have ? x : -kInf), uy = warp_maxf(have ? y : -kInf), uz = warp_maxf(have ? z : -kInf);
    if ((threadIdx.x & 31) == 0) {
        float *b = box + (threadIdx.x >> 5) * 6;
        b[0] = lx; b[1] = ly; b[2] = lz;
        b[3] = ux; b[4] = uy; b[5] = uz;
    }
}

}  // namespace gtd

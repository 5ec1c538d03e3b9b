// Hand-written adjoint of the FP64 leapfrog KDK direct-summation evolve: gradients of a loss on
// the final state with respect to the initial positions, velocities and masses.  There is no
// counterpart in the reference; the forward it differentiates is gtd::system::evolve(leapfrog_kdk)
// (gregsys.hpp:2946-2990, force gregsys.hpp:352-357).
//
// Forward, as a sequence of kicks K(c, x): v += c a(x) and drifts D: x += h v:
//     K(h/2, x0) D K(h, x1) D ... D K(h, x_{T-1}) D K(h/2, xT)
// (a step's closing half kick and the next step's opening half kick act at the same positions and
// merge into one full kick).  Reverse sweep from (lx, lv) = (dL/dxT, dL/dvT), mu = 0:
//     for k = T .. 0:   lx += c_k J(x_k)^T lv ;  mu += c_k (da/dm)^T lv ;  if k > 0: lv += h lx
// with, for a_i = sum_j G m_j d_ij / r^3 (d_ij = x_j - x_i),
//     (J^T w)_k = sum_j G [ u / r^3 - 3 d (d . u) / r^5 ],  u = m_k w_j - m_j w_k,  d = x_j - x_k
//     (dL/dm)_k += sum_j G (w_j . (x_k - x_j)) / r^3.
// Memory: by default the forward keeps every position (32 bytes per body and step) while they fit
// kKeepBytes, so the reverse sweep evaluates no force at all; otherwise, and whenever the caller names an
// interval C, it keeps (x_k, x_{k+1}, v_{k+1/2}) every C steps and the reverse sweep recomputes one
// segment of positions at a time from there.  Force and VJP both evaluate each unordered pair once;
// systems of a few thousand bodies take one launch per step each way.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <new>
#include <type_traits>

#include "direct_sym_reduce.cuh"
#include "gtd_internal.cuh"
#include "gtd_math.cuh"

namespace gtd {

// ---- the VJP of one force evaluation ----------------------------------------------------------
// With d = x_j - x_k, u = m_k w_j - m_j w_k:
//     T = [u - 3 d (d . u) / r^2] / r^3,   (J^T w)_k += G T,   (J^T w)_j -= G T
//     (dL/dm)_k += -G (w_j . d) / r^3,     (dL/dm)_j += G (w_k . d) / r^3
// d . u comes from the two products the mass terms need, and the factor 3 from masses scaled once per
// body: 39 FP64 operations per unordered pair for both bodies' four sums.
//
// Decomposition, column rotation and partial sums as in direct_sym.cu, with four words per body
// ((J^T w) and the mass term).
struct VjpArgs {
    SymGeom g;
    const double4 *x;  // positions + mass
    const double4 *w;  // c_k * lambda_v (xyz)
    double *rowpart, *colpart;
    int64_t unit0, unit1, col0;
    unsigned *queue;
};

struct VjpSums {  // (J^T w) / G and the mass term / G of one body over its partners
    double x, y, z, m;
    __device__ __forceinline__ void clear() { x = y = z = m = 0.0; }
};

// The pair of body k with body j, added to k's sums and (kSym) to j's.  kGuard: r2 may vanish.
template <bool kSym, bool kGuard>
__device__ __forceinline__ void vjp_pair(const double4 &xk, const double4 &wk, double m3k, double xj, double yj, double zj,
                                         double mj, double wjx, double wjy, double wjz, double m3j, VjpSums &k,
                                         VjpSums &j) {
    const double dx = xj - xk.x, dy = yj - xk.y, dz = zj - xk.z;
    const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
    double inv = inv_r(r2);
    if (kGuard) inv = r2 > 0.0 ? inv : 0.0;  // the body itself and padding contribute nothing
    const double inv2 = inv * inv, inv3 = inv2 * inv;
    const double A = fma(wjz, dz, fma(wjy, dy, wjx * dx)), B = fma(wk.z, dz, fma(wk.y, dy, wk.x * dx));
    const double c = inv2 * fma(m3k, A, -m3j * B);
    const double vx = fma(-c, dx, fma(xk.w, wjx, -mj * wk.x));
    const double vy = fma(-c, dy, fma(xk.w, wjy, -mj * wk.y));
    const double vz = fma(-c, dz, fma(xk.w, wjz, -mj * wk.z));
    k.x = fma(inv3, vx, k.x);
    k.y = fma(inv3, vy, k.y);
    k.z = fma(inv3, vz, k.z);
    k.m = fma(-A, inv3, k.m);
    if (kSym) {
        j.x = fma(-inv3, vx, j.x);
        j.y = fma(-inv3, vy, j.y);
        j.z = fma(-inv3, vz, j.z);
        j.m = fma(B, inv3, j.m);
    }
}

template <int T, int TC>
struct VjpSmem {
    static constexpr int kWarps = T / 32;
    // staged columns, each chunk of 32 twice in a row: (x, y), (z, m), (wx, wy), (wz, 3 m)
    double2 xy[2][TC / 32 * 64], zm[2][TC / 32 * 64], wxy[2][TC / 32 * 64], wz[2][TC / 32 * 64];
    double col[2][kWarps][4][TC];
    int64_t su[4];
};

template <int I, int T, int TC, int MINB, int U>
__global__ void __launch_bounds__(T, MINB) vjp_kernel(VjpArgs a) {
    using Smem = VjpSmem<T, TC>;
    constexpr int kChunks = TC / 32, kWarps = Smem::kWarps;
    static_assert(TC <= T, "a thread stages at most one column");
    extern __shared__ __align__(16) unsigned char vjp_smem[];
    Smem &S = *reinterpret_cast<Smem *>(vjp_smem);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
    auto stage = [&](int buf, const double4 &x, const double4 &w) {
        const int e = (t >> 5) * 64 + lane;
        S.xy[buf][e] = S.xy[buf][e + 32] = make_double2(x.x, x.y);
        S.zm[buf][e] = S.zm[buf][e + 32] = make_double2(x.z, x.w);
        S.wxy[buf][e] = S.wxy[buf][e + 32] = make_double2(w.x, w.y);
        S.wz[buf][e] = S.wz[buf][e + 32] = make_double2(w.z, 3.0 * x.w);
    };
    // padding columns: massless, weightless and far away (1 / r^3 underflows to 0)
    const double4 far = make_double4(1e120, 1e120, 1e120, 0.0), zero = make_double4(0.0, 0.0, 0.0, 0.0);
    for (;;) {
        if (t == 0) {
            const int64_t u = a.unit0 + (int64_t)atomicAdd(a.queue, 1u);
            S.su[0] = u;
            if (u < a.unit1) {
                const SymUnit o = sym_unit(a.g, u);
                S.su[1] = o.r;
                S.su[2] = o.c0;
                S.su[3] = o.c1;
            }
        }
        __syncthreads();
        const int64_t u = S.su[0];
        if (u >= a.unit1) break;
        const int64_t r = S.su[1], c0 = S.su[2], c1 = S.su[3], row0 = r * a.g.B;
        if (row0 >= a.g.n) {
            __syncthreads();
            continue;
        }
        double4 xk[I], wk[I];
        double m3[I];
        VjpSums row[I];
#pragma unroll
        for (int k = 0; k < I; ++k) {
            const int64_t i = row0 + k * T + t;
            xk[k] = i < a.g.n ? a.x[i] : zero;
            wk[k] = i < a.g.n ? a.w[i] : zero;
            m3[k] = 3.0 * xk[k].w;
            row[k].clear();
        }
        const int64_t own_end = (r / a.g.s + 1) * a.g.kw;
        const int64_t coff = sym_col_off(a.g, r) - a.col0 - own_end;
        const int64_t tail = a.g.n / 256 * (256 / TC);  // tiles of the last, incomplete 256 bodies: guarded as well
        if (c0 < c1 && t < TC) {
            const int64_t j = c0 * TC + t;
            stage(0, j < a.g.n ? a.x[j] : far, j < a.g.n ? a.w[j] : zero);
        }
        __syncthreads();
        int cur = 0;
        for (int64_t jt = c0; jt < c1; ++jt, cur ^= 1) {
            double4 xn = far, wn = zero;
            const bool more = jt + 1 < c1;
            if (more && t < TC) {
                const int64_t j = (jt + 1) * TC + t;
                if (j < a.g.n) {
                    xn = a.x[j];
                    wn = a.w[j];
                }
            }
            const bool sym = jt >= own_end;
            for (int ch = 0; ch < kChunks; ++ch) {
                const int base = ch * 64 + (sym ? lane : 0);
                const double2 *XY = S.xy[cur] + base, *ZM = S.zm[cur] + base, *WXY = S.wxy[cur] + base;
                const double2 *WZ = S.wz[cur] + base;
                VjpSums c;
                c.clear();
                if (sym) {
                    auto step = [&](auto guard, int s) {
                        const double2 xy = XY[s], zm = ZM[s], wxy = WXY[s], wz = WZ[s];
#pragma unroll
                        for (int k = 0; k < I; ++k)
                            vjp_pair<true, decltype(guard)::value>(xk[k], wk[k], m3[k], xy.x, xy.y, zm.x, zm.y, wxy.x, wxy.y,
                                                                   wz.x, wz.y, row[k], c);
                        c.x = __shfl_sync(0xffffffffu, c.x, lane + 1);
                        c.y = __shfl_sync(0xffffffffu, c.y, lane + 1);
                        c.z = __shfl_sync(0xffffffffu, c.z, lane + 1);
                        c.m = __shfl_sync(0xffffffffu, c.m, lane + 1);
                    };
                    if (jt >= tail) {
#pragma unroll 1
                        for (int s = 0; s < 32; ++s) step(std::true_type{}, s);
                    } else {
#pragma unroll U
                        for (int s = 0; s < 32; ++s) step(std::false_type{}, s);
                    }
                    double *o = &S.col[cur][warp][0][ch * 32 + lane];
                    o[0] = c.x;
                    o[TC] = c.y;
                    o[2 * TC] = c.z;
                    o[3 * TC] = c.m;
                } else {
#pragma unroll 1
                    for (int s = 0; s < 32; ++s) {
                        const double2 xy = XY[s], zm = ZM[s], wxy = WXY[s], wz = WZ[s];
#pragma unroll
                        for (int k = 0; k < I; ++k)
                            vjp_pair<false, true>(xk[k], wk[k], m3[k], xy.x, xy.y, zm.x, zm.y, wxy.x, wxy.y, wz.x, wz.y, row[k], c);
                    }
                }
            }
            if (more && t < TC) stage(cur ^ 1, xn, wn);
            __syncthreads();
            if (sym) {
                double *slot = a.colpart + (size_t)(coff + jt) * 4 * TC;
                const double *cs = &S.col[cur][0][0][0];
#pragma unroll
                for (int e = t; e < 4 * TC; e += T) slot[e] = sym_tree<kWarps>([&](int w) { return cs[w * 4 * TC + e]; });
            }
        }
        double *slot = a.rowpart + (size_t)(u - a.unit0) * 4 * a.g.B;
#pragma unroll
        for (int k = 0; k < I; ++k) {
            const int l = k * T + t;
            slot[l] = row[k].x;
            slot[a.g.B + l] = row[k].y;
            slot[2 * a.g.B + l] = row[k].z;
            slot[3 * a.g.B + l] = row[k].m;
        }
        __syncthreads();
    }
}

// lx += G J^T w ; mu += G (..) ; then (if drift) lv += h lx ; and w = c lv for the next VJP
struct VjpUpdate {
    double G, h;
    double4 *lx, *lv;
    double *mu;
    double4 *w_next;
    double c_next;
    int drift;
    __device__ __forceinline__ void apply(int64_t i, double jx, double jy, double jz, double m) const {
        double4 x = lx[i];
        x.x = fma(G, jx, x.x);
        x.y = fma(G, jy, x.y);
        x.z = fma(G, jz, x.z);
        lx[i] = x;
        mu[i] = fma(G, m, mu[i]);
        if (drift) {
            double4 v = lv[i];
            v.x = fma(h, x.x, v.x);
            v.y = fma(h, x.y, v.y);
            v.z = fma(h, x.z, v.z);
            lv[i] = v;
            w_next[i] = make_double4(c_next * v.x, c_next * v.y, c_next * v.z, 0.0);
        }
    }
};

// Small systems: VJP and update in one launch, as fused_small_kernel (direct.cu) does force and step.
// kVjpSlices warps share a body, their lanes take the ordered pairs of every 32 kVjpSlices-th partner
// straight from L1 / L2, and the body's first warp adds the slices in order.  Chained launches: a reverse
// step of 1000 bodies 8.8 -> 8.1 us (7.2 with two bodies per warp), of 2000 16.9 -> 15.2, with warp_sums 14.8.
constexpr int kVjpSlices = 4;

template <int I, int GROUPS, int MINB>
__global__ void __launch_bounds__(GROUPS * kVjpSlices * 32, MINB)
    vjp_small_kernel(int64_t n, const double4 *x, const double4 *w, VjpUpdate up) {
    __shared__ double part[kVjpSlices][GROUPS][I][4];
    cudaGridDependencySynchronize();
    const int wp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int bl = wp % GROUPS, slice = wp / GROUPS;
    const int64_t i0 = ((int64_t)blockIdx.x * GROUPS + bl) * I;
    double4 xk[I], wk[I];
    VjpSums s[I], none;
#pragma unroll
    for (int k = 0; k < I; ++k) {
        xk[k] = i0 + k < n ? x[i0 + k] : make_double4(0.0, 0.0, 0.0, 0.0);
        wk[k] = i0 + k < n ? w[i0 + k] : make_double4(0.0, 0.0, 0.0, 0.0);
        s[k].clear();
    }
    if (i0 < n) {
#pragma unroll 2
        for (int64_t j = (int64_t)slice * 32 + lane; j < n; j += 32 * kVjpSlices) {
            const double4 xj = x[j], wj = w[j];
#pragma unroll
            for (int k = 0; k < I; ++k)
                vjp_pair<false, true>(xk[k], wk[k], 3.0 * xk[k].w, xj.x, xj.y, xj.z, xj.w, wj.x, wj.y, wj.z, 3.0 * xj.w, s[k],
                                      none);
        }
    }
    cudaTriggerProgrammaticLaunchCompletion();
    double sums[4 * I];
#pragma unroll
    for (int k = 0; k < I; ++k) {
        sums[4 * k] = s[k].x;
        sums[4 * k + 1] = s[k].y;
        sums[4 * k + 2] = s[k].z;
        sums[4 * k + 3] = s[k].m;
    }
    int at;
    const double sum = warp_sums(sums, at);
    if (at >= 0) (&part[slice][bl][0][0])[at] = sum;
    __syncthreads();
    if (slice == 0 && lane < I && i0 + lane < n) {
        double v[4];
#pragma unroll
        for (int d = 0; d < 4; ++d) {
            v[d] = part[0][bl][lane][d];
#pragma unroll
            for (int k = 1; k < kVjpSlices; ++k) v[d] += part[k][bl][lane][d];
        }
        up.apply(i0 + lane, v[0], v[1], v[2], v[3]);
    }
}

template <int I, int GROUPS, int MINB>
static void launch_vjp_small(int64_t n, const double4 *x, const double4 *w, const VjpUpdate &up, cudaStream_t st) {
    launch_chained(true, vjp_small_kernel<I, GROUPS, MINB>, (unsigned)((n + GROUPS * I - 1) / (GROUPS * I)),
                   GROUPS * kVjpSlices * 32, 0, st, n, x, w, up);
}

__global__ void __launch_bounds__(kRedWarps * 32) vjp_reduce_kernel(SymSlots s, double *base_out, VjpUpdate up,
                                                                    unsigned *queue) {
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
    if (blockIdx.x == 0 && threadIdx.x == 0) *queue = 0;  // the batch's counter, for the next VJP
    sym_reduce<4>(s, [&](int64_t i, const double (&v)[4]) {
        if (base_out) {  // not the last batch
#pragma unroll
            for (int d = 0; d < 4; ++d) base_out[(size_t)d * s.g.n + i] = v[d];
        } else {
            up.apply(i, v[0], v[1], v[2], v[3]);
        }
    });
}

// Two rows per thread, 3 CTAs per SM: 0.43 ms at N = 16384, 69 % of the FP64 pipe (the form with 47
// operations and a thread per body for the sums: 0.53).  Eight sums per body with u never formed (39
// operations too) ran at 0.48 ms: twice the shuffles.  Four rows per thread: 240 registers, no faster.
constexpr SymShape kVjpShape{2, 128, 64, 256};
constexpr size_t kVjpSmem = sizeof(VjpSmem<128, 64>);
static constexpr auto kVjpKernel = vjp_kernel<2, 128, 64, 3, 2>;

__global__ void pack_kernel(int64_t n, const double *x3, const double *m, const double *v3, double4 *x, double4 *v) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    x[i] = make_double4(x3[3 * i], x3[3 * i + 1], x3[3 * i + 2], m[i]);
    if (v) v[i] = make_double4(v3[3 * i], v3[3 * i + 1], v3[3 * i + 2], 0.0);
}

__global__ void unpack_kernel(int64_t n, const double4 *a, double *a3) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double4 q = a[i];
    a3[3 * i] = q.x;
    a3[3 * i + 1] = q.y;
    a3[3 * i + 2] = q.z;
}

// The reverse sweep's start: lx = gx, lv = gv (0 where NULL), mu = 0, w = c lv
__global__ void reverse_begin_kernel(int64_t n, const double *gx, const double *gv, double c, double4 *lx, double4 *lv,
                                     double *mu, double4 *w) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    lx[i] = make_double4(gx[3 * i], gx[3 * i + 1], gx[3 * i + 2], 0.0);
    const double4 v = gv ? make_double4(gv[3 * i], gv[3 * i + 1], gv[3 * i + 2], 0.0) : make_double4(0, 0, 0, 0);
    lv[i] = v;
    mu[i] = 0.0;
    w[i] = make_double4(c * v.x, c * v.y, c * v.z, 0.0);
}

}  // namespace gtd

using namespace gtd;

struct gtd_adjoint {
    int device = 0;
    int64_t n = 0;
    uint64_t steps = 0, every = 0;  // every == 0: all positions are kept
    double G = 0, h = 0;
    ForcePlan fplan;
    SymGeom vgeom;
    int vgrid = 0;
    bool small_force = false, small_vjp = false;
    char *mem = nullptr;  // every buffer below
    bool owned = false;
    double4 *pos = nullptr;   // all positions [(steps + 1) n], or two buffers in turn
    double4 *v = nullptr;
    double4 *ck = nullptr;    // checkpoints: (x_k, x_{k+1}, v_{k+1/2}) each
    double4 *seg = nullptr;   // positions of one segment [(every + 1) n]
    double4 *lx = nullptr, *lv = nullptr, *w[2] = {nullptr, nullptr};
    double *mu = nullptr, *fpart = nullptr, *vpart = nullptr;
    bool have_forward = false;
    uint64_t launches = 0;
};

static unsigned g1(int64_t n) { return (unsigned)((n + 255) / 256); }

// Bytes of positions that the forward keeps rather than recompute them: 16384 bodies over 2000 steps.
constexpr size_t kKeepBytes = (size_t)5 << 28;
// Up to this many bodies a VJP and its update run as one launch: 17 us a step at N = 2048 (31 in the
// blocked form), 31 at 3000 (40), 39 at 3500 (41).
constexpr int64_t kVjpSmallMaxN = 3400;

// Fills the plan and lays the buffers out from `base` (sizes only where base is NULL); the bytes they take.
static size_t adj_layout(gtd_adjoint *A, char *base) {
    const int64_t n = A->n;
    const size_t b4 = sizeof(double4) * (size_t)n;
    size_t at = 0;
    auto take = [&](auto *&p, size_t bytes) {
        p = base ? reinterpret_cast<std::remove_reference_t<decltype(p)>>(base + at) : nullptr;
        at += (bytes + 255) / 256 * 256;
    };
    take(A->pos, b4 * (size_t)(A->every ? 2 : A->steps + 1));
    take(A->v, b4);
    if (A->every) {
        take(A->ck, 3 * b4 * (size_t)((A->steps + A->every - 1) / A->every));
        take(A->seg, b4 * (size_t)(A->every + 1));
    }
    take(A->lx, b4);
    take(A->lv, b4);
    take(A->w[0], b4);
    take(A->w[1], b4);
    take(A->mu, sizeof(double) * (size_t)n);
    if (!A->small_force) take(A->fpart, partial_bytes(A->fplan));
    if (!A->small_vjp) take(A->vpart, sym_layout(A->vgeom, kSymSlotBytes, 4).bytes);
    return at;
}

static int adj_new(gtd_adjoint **out, int device, int64_t n, uint64_t steps, uint64_t checkpoint_every, double G,
                   double dt) {
    *out = nullptr;
    if (n < 2 || steps < 1 || !(dt > 0)) return fail(GTD_ERR_INVALID_ARGUMENT, "need n >= 2, steps >= 1, dt > 0");
    GTD_CUDA(cudaSetDevice(device));
    gtd_adjoint *A = new (std::nothrow) gtd_adjoint();
    if (!A) return fail(GTD_ERR_OUT_OF_MEMORY, "host allocation failed");
    A->device = device;
    A->n = n;
    A->steps = steps;
    A->every = std::min<uint64_t>(checkpoint_every, steps);
    if (checkpoint_every == 0 && steps >= kKeepBytes / (sizeof(double4) * (size_t)n))
        A->every = std::max<uint64_t>(1, (uint64_t)std::llround(std::sqrt((double)steps)));
    A->G = G;
    A->h = dt;
    A->small_force = n <= kFusedAutoMaxN;
    A->small_vjp = n <= kVjpSmallMaxN;
    if (!A->small_force) A->fplan = make_plan(n, GTD_PREC_F64, device, tuned_variant(device, GTD_PREC_F64, n));
    if (!A->small_vjp) {
        int sms = 148, per_sm = 1;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        cudaFuncSetAttribute(kVjpKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kVjpSmem);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kVjpKernel, kVjpShape.threads, kVjpSmem);
        per_sm = std::max(per_sm, 1);
        A->vgeom = sym_geometry(n, kVjpShape, sms, per_sm);
        A->vgrid = sms * per_sm;
    }
    *out = A;
    return GTD_OK;
}

// The force at src, v += c a and, unless dst is NULL, dst = src + h v.
static int adj_step(gtd_adjoint *A, const double4 *src, double4 *dst, double c, cudaStream_t st) {
    StepArgs sa{};
    sa.n = A->n;
    sa.src = sa.cur = src;
    sa.dst = dst;
    sa.vel = A->v;
    sa.h = A->h;
    sa.hp = c;
    sa.last = dst ? 0 : 1;
    if (A->small_force) {
        A->launches += 1;
        return launch_fused_small(A->n, src, A->G, EPI_KICK_DRIFT, sa, st, true);
    }
    int rc = launch_force(GTD_PREC_F64, A->fplan, src, A->G, A->fpart, st, true);
    if (!rc) rc = launch_integrate(A->fplan, A->fpart, EPI_KICK_DRIFT, sa, st, true);
    A->launches += (uint64_t)force_launch_count(A->fplan);
    return rc;
}

// The queue counters of the pair kernels, zero before a sweep; each reduction restores its own.
static int adj_reset(gtd_adjoint *A, cudaStream_t st) {
    if (!A->small_force && A->fplan.sym) {
        const int rc = sym_reset(A->fplan, A->fpart, st);
        if (rc) return rc;
    }
    if (!A->small_vjp)
        GTD_CUDA(cudaMemsetAsync(A->vpart, 0, (size_t)sym_layout(A->vgeom, kSymSlotBytes, 4).batches * sizeof(unsigned), st));
    return GTD_OK;
}

// The VJP at x_k with w = c_k lv, and the update; w for x_{k-1} is left in the other buffer.
static int adj_vjp(gtd_adjoint *A, const double4 *x, uint64_t k, int &cur, cudaStream_t st) {
    const VjpUpdate up{A->G, A->h, A->lx, A->lv, A->mu, A->w[cur ^ 1], k == 1 ? 0.5 * A->h : A->h, k > 0 ? 1 : 0};
    const double4 *w = A->w[cur];
    cur ^= 1;
    if (A->small_vjp) {
        // bodies per warp, CTAs per SM and the sizes where they change as in launch_fused_small, up to two
        // bodies.  Us a step both ways with one body per warp and two: 500 bodies 7.49 / 7.82, 592 8.45 /
        // 8.43, 700 9.14 / 9.18, 800 10.0 / 9.28, 1000 11.8 / 10.9, 1184 13.3 / 13.0, 1480 21.1 / 15.2
        if (A->n <= 592) launch_vjp_small<1, 1, 8>(A->n, x, w, up, st);
        else if (A->n <= 5 * 148 * 2) launch_vjp_small<2, 1, 5>(A->n, x, w, up, st);
        else launch_vjp_small<2, 1, 4>(A->n, x, w, up, st);
        GTD_CHECK_LAUNCH();
        A->launches += 1;
        return GTD_OK;
    }
    const SymGeom &g = A->vgeom;
    const SymLayout lay = sym_layout(g, kSymSlotBytes, 4);
    char *mem = reinterpret_cast<char *>(A->vpart);
    int64_t batch = 0;
    for (int64_t Pa = 0; Pa < g.Gs; ++batch) {
        const int64_t Pb = sym_batch_end(g, Pa, kSymSlotBytes, 4);
        const SymSlots s = sym_slots(g, lay, mem, Pa, Pb, 4);
        const VjpArgs va{g, x, w, const_cast<double *>(s.rowpart), const_cast<double *>(s.colpart), s.unit0,
                         sym_tri(g, Pb) * sym_block_units(g), s.col0, reinterpret_cast<unsigned *>(mem) + batch};
        const int grid = (int)std::min<int64_t>(A->vgrid, va.unit1 - va.unit0);
        launch_chained(true, kVjpKernel, grid, kVjpShape.threads, kVjpSmem, st, va);
        GTD_CHECK_LAUNCH();
        double *base = Pb < g.Gs ? reinterpret_cast<double *>(mem + lay.base) : nullptr;
        launch_chained(true, vjp_reduce_kernel, (unsigned)((g.n + 31) / 32), kRedWarps * 32, 0, st, s, base, up, va.queue);
        GTD_CHECK_LAUNCH();
        A->launches += 2;
        Pa = Pb;
    }
    return GTD_OK;
}

extern "C" {

int gtd_adjoint_create(gtd_adjoint **out, int device, int64_t n, uint64_t steps, uint64_t checkpoint_every,
                       double G, double dt) {
    if (!out) return fail(GTD_ERR_INVALID_ARGUMENT, "out is NULL");
    gtd_adjoint *A = nullptr;
    int rc = adj_new(&A, device, n, steps, checkpoint_every, G, dt);
    if (rc) return rc;
    const cudaError_t e = cudaMalloc((void **)&A->mem, adj_layout(A, nullptr));
    if (e != cudaSuccess) {
        rc = cuda_fail(e, "adjoint buffers", __FILE__, __LINE__);
        delete A;
        return rc;
    }
    A->owned = true;
    adj_layout(A, A->mem);
    *out = A;
    return GTD_OK;
}

int gtd_adjoint_workspace_bytes(int device, int64_t n, uint64_t steps, uint64_t checkpoint_every, uint64_t *bytes) {
    if (!bytes) return fail(GTD_ERR_INVALID_ARGUMENT, "bytes is NULL");
    *bytes = 0;
    gtd_adjoint *A = nullptr;
    int rc = adj_new(&A, device, n, steps, checkpoint_every, 1.0, 1.0);
    if (rc) return rc;
    *bytes = adj_layout(A, nullptr);
    delete A;
    return GTD_OK;
}

int gtd_adjoint_create_in(gtd_adjoint **out, int device, int64_t n, uint64_t steps, uint64_t checkpoint_every,
                          double G, double dt, void *workspace, uint64_t bytes) {
    if (!out) return fail(GTD_ERR_INVALID_ARGUMENT, "out is NULL");
    *out = nullptr;
    if (!workspace || reinterpret_cast<uintptr_t>(workspace) % 256 != 0)
        return fail(GTD_ERR_INVALID_ARGUMENT, "the workspace must be 256-byte aligned device memory");
    gtd_adjoint *A = nullptr;
    int rc = adj_new(&A, device, n, steps, checkpoint_every, G, dt);
    if (rc) return rc;
    const size_t need = adj_layout(A, nullptr);
    if (need > bytes) {
        delete A;
        return fail(GTD_ERR_CAPACITY, "the adjoint needs a workspace of %zu bytes, got %llu", need,
                    (unsigned long long)bytes);
    }
    A->mem = static_cast<char *>(workspace);
    adj_layout(A, A->mem);
    *out = A;
    return GTD_OK;
}

int gtd_adjoint_destroy(gtd_adjoint *A) {
    if (!A) return GTD_OK;
    if (A->owned) {
        cudaSetDevice(A->device);
        cudaFree(A->mem);
    }
    delete A;
    return GTD_OK;
}

// Forward KDK over all steps from device arrays x0/v0 (n x 3) and m (n); writes xT/vT (device, may
// be NULL) and keeps what gtd_adjoint_backward needs.  stream: a cudaStream_t or NULL.
int gtd_adjoint_forward(gtd_adjoint *A, const double *x0, const double *v0, const double *m, double *xT,
                        double *vT, void *stream) {
    if (!A || !x0 || !v0 || !m) return fail(GTD_ERR_INVALID_ARGUMENT, "NULL argument");
    GTD_CUDA(cudaSetDevice(A->device));
    cudaStream_t st = (cudaStream_t)stream;
    const int64_t n = A->n;
    const size_t b4 = sizeof(double4) * (size_t)n;
    const uint64_t T = A->steps, C = A->every;
    const double h = A->h;
    int rc = adj_reset(A, st);
    if (rc) return rc;
    auto at = [&](uint64_t k) { return A->pos + (size_t)(C ? k & 1 : k) * (size_t)n; };
    pack_kernel<<<g1(n), 256, 0, st>>>(n, x0, m, v0, at(0), A->v);
    GTD_CHECK_LAUNCH();
    A->launches += 1;
    for (uint64_t k = 0; k <= T; ++k) {
        rc = adj_step(A, at(k), k < T ? at(k + 1) : nullptr, k == 0 || k == T ? 0.5 * h : h, st);
        if (rc) return rc;
        if (C && k < T && k % C == 0) {
            double4 *c = A->ck + 3 * (size_t)n * (size_t)(k / C);
            GTD_CUDA(cudaMemcpyAsync(c, at(k), b4, cudaMemcpyDeviceToDevice, st));
            GTD_CUDA(cudaMemcpyAsync(c + n, at(k + 1), b4, cudaMemcpyDeviceToDevice, st));
            GTD_CUDA(cudaMemcpyAsync(c + 2 * n, A->v, b4, cudaMemcpyDeviceToDevice, st));
        }
    }
    if (xT) unpack_kernel<<<g1(n), 256, 0, st>>>(n, at(T), xT);
    if (vT) unpack_kernel<<<g1(n), 256, 0, st>>>(n, A->v, vT);
    GTD_CHECK_LAUNCH();
    A->have_forward = true;
    return GTD_OK;
}

// Reverse sweep: gxT, gvT (device, n x 3, gvT may be NULL) -> gx0, gv0 (n x 3), gm (n).
int gtd_adjoint_backward(gtd_adjoint *A, const double *gxT, const double *gvT, double *gx0, double *gv0, double *gm,
                         void *stream) {
    if (!A || !gxT) return fail(GTD_ERR_INVALID_ARGUMENT, "NULL argument");
    if (!A->have_forward) return fail(GTD_ERR_INVALID_ARGUMENT, "gtd_adjoint_forward must run first");
    GTD_CUDA(cudaSetDevice(A->device));
    cudaStream_t st = (cudaStream_t)stream;
    const int64_t n = A->n;
    const size_t b4 = sizeof(double4) * (size_t)n;
    const double h = A->h;
    const uint64_t T = A->steps, C = A->every;
    int cur = 0;
    {
        const int rc = adj_reset(A, st);
        if (rc) return rc;
    }
    reverse_begin_kernel<<<g1(n), 256, 0, st>>>(n, gxT, gvT, 0.5 * h, A->lx, A->lv, A->mu, A->w[0]);
    GTD_CHECK_LAUNCH();
    A->launches += 1;
    if (!C) {
        for (uint64_t k = T + 1; k-- > 0;) {
            const int rc = adj_vjp(A, A->pos + (size_t)k * (size_t)n, k, cur, st);
            if (rc) return rc;
        }
    } else {
        const int64_t nseg = (int64_t)((T + C - 1) / C);
        for (int64_t sgi = nseg - 1; sgi >= 0; --sgi) {
            const uint64_t k0 = (uint64_t)sgi * C, k1 = std::min<uint64_t>(k0 + C, T);
            // recompute positions x_{k0..k1} of this segment from its checkpoint
            const double4 *c = A->ck + 3 * (size_t)n * (size_t)sgi;
            GTD_CUDA(cudaMemcpyAsync(A->seg, c, 2 * b4, cudaMemcpyDeviceToDevice, st));
            GTD_CUDA(cudaMemcpyAsync(A->v, c + 2 * n, b4, cudaMemcpyDeviceToDevice, st));
            for (uint64_t k = k0 + 1; k < k1; ++k) {
                double4 *x = A->seg + (size_t)(k - k0) * (size_t)n;
                const int rc = adj_step(A, x, x + n, h, st);
                if (rc) return rc;
            }
            // VJPs at x_k, k = k1 .. k0 + 1, and at x_0 with the first segment
            const uint64_t kstop = sgi == 0 ? k0 : k0 + 1;
            for (uint64_t k = k1 + 1; k-- > kstop;) {
                const int rc = adj_vjp(A, A->seg + (size_t)(k - k0) * (size_t)n, k, cur, st);
                if (rc) return rc;
            }
        }
    }
    if (gx0) unpack_kernel<<<g1(n), 256, 0, st>>>(n, A->lx, gx0);
    if (gv0) unpack_kernel<<<g1(n), 256, 0, st>>>(n, A->lv, gv0);
    if (gm) GTD_CUDA(cudaMemcpyAsync(gm, A->mu, sizeof(double) * (size_t)n, cudaMemcpyDeviceToDevice, st));
    GTD_CHECK_LAUNCH();
    return GTD_OK;
}

int gtd_adjoint_launch_count(const gtd_adjoint *A, uint64_t *count) {
    if (!A || !count) return fail(GTD_ERR_INVALID_ARGUMENT, "NULL argument");
    *count = A->launches;
    return GTD_OK;
}

}  // extern "C"

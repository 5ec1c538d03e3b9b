// Direct-summation force kernels that evaluate each unordered pair once.
//
// The force of a pair is antisymmetric up to the two masses: with d = x_j - x_i, body i receives
// G m_j d / r^3 and body j receives -G m_i d / r^3.  Per unordered pair that is 17 FP32 (20 FP64)
// lane-operations for both bodies, against 2 x 12 (2 x 16) when every ordered pair is evaluated by
// itself (cumulative_acc, gregsys.hpp:352-357, direct.cu); both kernels are bound by their FMA pipe.
//
// Work.  The bodies are cut into groups of W consecutive bodies, groups into row blocks of B (the
// bodies a CTA holds in registers, I per thread) and into column tiles of TC (staged in shared
// memory).  A unit is one row block against a run of column tiles that start at or after the row
// block's own group.  Tiles of the row block's own group are summed as ordered pairs, for the rows
// alone, with the self pair and coincident bodies selected away; every later tile is summed once for
// rows and columns.  Units are taken in turn from a counter, so CTAs with cheaper units take more.
//
// Rows are summed in registers; a unit writes one row sum per body.  Columns: inside a chunk of 32
// (packed) columns lane l pairs its rows with column (l + s) mod 32 at step s and carries that
// column's running sum, which one shuffle per component passes on to lane l - 1 after the step.  The
// warps' column sums meet in shared memory and are added in FP64, in warp order, into one slot per
// (row block, tile).  sym_reduce_kernel adds a body's row and column slots in a fixed order: the
// results do not depend on which CTA took which unit, and are bit-reproducible.
//
// The column slots take 24 N^2 / (2 B) bytes.  Where that exceeds the plan's bound the row groups are
// processed in batches, each reduced into a running sum before the next reuses the slots.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <type_traits>

#include "direct_epilogue.cuh"
#include "direct_mixed.cuh"
#include "direct_sym_reduce.cuh"
#include "gtd_internal.cuh"
#include "gtd_math.cuh"

namespace gtd {

struct SymKArgs {
    SymGeom g;
    const double4 *src;
    double G;
    double *rowpart, *colpart;  // slots of this batch
    int64_t unit0, unit1;       // units of this batch
    int64_t col0;               // first column slot of this batch
    float near2;
    unsigned *queue;            // zero before the launch
};

// -------------------------------------------------------------------------------------------
// FP64
// -------------------------------------------------------------------------------------------
template <int I, int T, int TC, int MINB>
__global__ void __launch_bounds__(T, MINB) force_f64_sym_kernel(SymKArgs a) {
    constexpr int kWarps = T / 32, kChunks = TC / 32;
    // (x, y) and (z, G m) of the staged columns; each chunk of 32 is stored twice in a row, so that
    // the column (l + s) mod 32 is entry l + s
    __shared__ double2 sxy[2][kChunks * 64], szm[2][kChunks * 64];
    __shared__ double col[2][kWarps][3][TC];
    __shared__ int64_t su[4];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
    auto stage = [&](int buf, int c, const double4 &q) {
        const int e = (c >> 5) * 64 + (c & 31);
        sxy[buf][e] = sxy[buf][e + 32] = make_double2(q.x, q.y);
        szm[buf][e] = szm[buf][e + 32] = make_double2(q.z, q.w);
    };
    auto fetch = [&](int64_t j) {  // padding columns: massless and far away (r^-3 underflows to 0)
        double4 q = make_double4(1e150, 1e150, 1e150, 0.0);
        if (j < a.g.n) {
            q = a.src[j];
            q.w *= a.G;
        }
        return q;
    };
    for (;;) {
        if (t == 0) {
            const int64_t u = a.unit0 + (int64_t)atomicAdd(a.queue, 1u);
            su[0] = u;
            if (u < a.unit1) {
                const SymUnit o = sym_unit(a.g, u);
                su[1] = o.r;
                su[2] = o.c0;
                su[3] = o.c1;
            }
        }
        __syncthreads();
        const int64_t u = su[0];
        if (u >= a.unit1) break;
        const int64_t r = su[1], c0 = su[2], c1 = su[3];
        const int64_t row0 = r * a.g.B;
        if (row0 >= a.g.n) {  // the last group's missing row blocks
            __syncthreads();
            continue;
        }
        double xi[I], yi[I], zi[I], mi[I], ax[I], ay[I], az[I];
#pragma unroll
        for (int k = 0; k < I; ++k) {
            const int64_t i = row0 + k * T + t;
            const double4 p = i < a.g.n ? a.src[i] : make_double4(0.0, 0.0, 0.0, 0.0);
            xi[k] = p.x; yi[k] = p.y; zi[k] = p.z; mi[k] = p.w * a.G;
            ax[k] = ay[k] = az[k] = 0.0;
        }
        const int64_t own_end = (r / a.g.s + 1) * a.g.kw;  // tiles below are ordered pairs
        const int64_t coff = sym_col_off(a.g, r) - a.col0 - own_end;
        // Coincident bodies: selected away within the row block's group and in the last, incomplete 256
        // bodies, where the ordered-pair kernel does so too.
        const int64_t tail = a.g.n / 256 * (256 / TC);
        if (c0 < c1)
            for (int c = t; c < TC; c += T) stage(0, c, fetch(c0 * TC + c));
        __syncthreads();
        int cur = 0;
        for (int64_t jt = c0; jt < c1; ++jt, cur ^= 1) {
            constexpr int kFetch = (TC + T - 1) / T;
            double4 qn[kFetch];
            const bool more = jt + 1 < c1;
#pragma unroll
            for (int f = 0; f < kFetch; ++f)
                if (more && t + f * T < TC) qn[f] = fetch((jt + 1) * TC + t + f * T);
            const bool sym = jt >= own_end;
            if (sym) {
                for (int ch = 0; ch < kChunks; ++ch) {
                    const double2 *XY = sxy[cur] + ch * 64 + lane, *ZM = szm[cur] + ch * 64 + lane;
                    double cx = 0.0, cy = 0.0, cz = 0.0;
                    auto step = [&](auto guard, int s) {
                        const double2 xy = XY[s], zm = ZM[s];
#pragma unroll
                        for (int k = 0; k < I; ++k) {
                            const double dx = xy.x - xi[k], dy = xy.y - yi[k], dz = zm.x - zi[k];
                            const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
                            double w = inv_r3(r2);
                            if (decltype(guard)::value) w = r2 > 0.0 ? w : 0.0;
                            const double sj = zm.y * w, si = mi[k] * w;
                            ax[k] = fma(sj, dx, ax[k]);
                            ay[k] = fma(sj, dy, ay[k]);
                            az[k] = fma(sj, dz, az[k]);
                            cx = fma(si, dx, cx);
                            cy = fma(si, dy, cy);
                            cz = fma(si, dz, cz);
                        }
                        cx = __shfl_sync(0xffffffffu, cx, lane + 1);
                        cy = __shfl_sync(0xffffffffu, cy, lane + 1);
                        cz = __shfl_sync(0xffffffffu, cz, lane + 1);
                    };
                    if (jt >= tail) {
#pragma unroll 1
                        for (int s = 0; s < 32; ++s) step(std::true_type{}, s);
                    } else {
#pragma unroll 4
                        for (int s = 0; s < 32; ++s) step(std::false_type{}, s);
                    }
                    col[cur][warp][0][ch * 32 + lane] = cx;
                    col[cur][warp][1][ch * 32 + lane] = cy;
                    col[cur][warp][2][ch * 32 + lane] = cz;
                }
            } else {
                for (int ch = 0; ch < kChunks; ++ch) {
                    const double2 *XY = sxy[cur] + ch * 64, *ZM = szm[cur] + ch * 64;
#pragma unroll 4
                    for (int s = 0; s < 32; ++s) {
                        const double2 xy = XY[s], zm = ZM[s];
#pragma unroll
                        for (int k = 0; k < I; ++k) {
                            const double dx = xy.x - xi[k], dy = xy.y - yi[k], dz = zm.x - zi[k];
                            const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
                            const double w = zm.y * inv_r3(r2);
                            const double sj = r2 > 0.0 ? w : 0.0;
                            ax[k] = fma(sj, dx, ax[k]);
                            ay[k] = fma(sj, dy, ay[k]);
                            az[k] = fma(sj, dz, az[k]);
                        }
                    }
                }
            }
#pragma unroll
            for (int f = 0; f < kFetch; ++f)
                if (more && t + f * T < TC) stage(cur ^ 1, t + f * T, qn[f]);
            __syncthreads();
            if (sym) {
                double *slot = a.colpart + (size_t)(coff + jt) * 3 * TC;
                const double *cs = &col[cur][0][0][0];
#pragma unroll
                for (int e = t; e < 3 * TC; e += T) slot[e] = -sym_tree<kWarps>([&](int w) { return cs[w * 3 * TC + e]; });
            }
        }
        double *slot = a.rowpart + (size_t)(u - a.unit0) * 3 * a.g.B;
#pragma unroll
        for (int k = 0; k < I; ++k) {
            const int l = k * T + t;
            slot[l] = ax[k];
            slot[a.g.B + l] = ay[k];
            slot[2 * a.g.B + l] = az[k];
        }
        __syncthreads();  // orders every read of su before thread 0 takes the next unit
    }
}

// -------------------------------------------------------------------------------------------
// Mixed precision: FP32 pair terms in each row block's own frame, two columns per packed
// instruction, the close-pair precise path and the FP64 Kahan folds of direct.cu's kernel.  The FP32
// chains are no longer than there: a row folds after FC columns (FC / 2 terms per packed half), a
// column after 32 / NH steps (32 I / NH terms per packed half).
//
// Four rows per thread: a step's column reads (two 16-byte shared loads) and its six shuffles serve
// 8 pairs; at two rows they take as many cycles as the arithmetic.  The Kahan sums, touched once per
// fold, sit in shared memory, which leaves 168 registers per thread for 3 CTAs of 4 warps per SM.
// -------------------------------------------------------------------------------------------
template <int I, int T, int TC, int NH>
struct SymMixedSmem {
    static constexpr int kWarps = T / 32, kChunks = TC / 64;
    float4 xy[2][kChunks * 64], zm[2][kChunks * 64];  // (x x' y y'), (z z' Gm Gm') of packed columns, each chunk twice
    float2 lx[2][TC / 2], ly[2][TC / 2], lz[2][TC / 2];  // FP32 remainders of the coordinates
    float col[2][kWarps][NH][3][TC];                  // the warps' column sums, NH per chunk of 32 steps
    float ilo[3][I][T];                               // remainders of the rows' coordinates
    double kah[6][I][T];                              // FP64 Kahan sums of the rows
    float jbox[2][TC / 32][6];
    float ibox[kWarps][7];
    double cred[3][kWarps];
    int64_t su[4];
};

// One chunk of 64 columns (32 packed pairs).  kSym: rows and columns, lane l on packed column
// (l + s) mod 32 at step s.  Otherwise: rows alone, every lane on the same column.  The precise path
// takes its differences from the hi/lo splits.  A vanishing separation (the self pair, coincident
// bodies) is selected away wherever it can occur: on the ordered path, on the precise one and (kGuard) in
// the guarded chunks of the kernel without the close-pair check.
template <int I, int T, int U, int NH, bool kSym, bool kPrecise, bool kGuard = kPrecise || !kSym>
__device__ __forceinline__ void sym_mixed_chunk(const float4 *xy, const float4 *zm, const float2 *lx, const float2 *ly,
                                                const float2 *lz, const float (*ilo)[I][T], const float2 (&nx)[I],
                                                const float2 (&ny)[I], const float2 (&nz)[I], const float2 (&mi)[I],
                                                float2 (&fx)[I], float2 (&fy)[I], float2 (&fz)[I],
                                                float *col, int tc) {
    const int t = threadIdx.x, lane = t & 31;
    float2 qx[I], qy[I], qz[I];
    if (kPrecise) {
#pragma unroll
        for (int k = 0; k < I; ++k) {
            const float x = -ilo[0][k][t], y = -ilo[1][k][t], z = -ilo[2][k][t];
            qx[k] = make_float2(x, x);
            qy[k] = make_float2(y, y);
            qz[k] = make_float2(z, z);
        }
    }
    const float4 *XY = xy + (kSym ? lane : 0), *ZM = zm + (kSym ? lane : 0);
#pragma unroll 1
    for (int part = 0; part < NH; ++part) {
        constexpr int kSteps = 32 / NH;
        float2 cx = make_float2(0.f, 0.f), cy = cx, cz = cx;
#pragma unroll U
        for (int s = 0; s < kSteps; ++s) {
            const float4 A = XY[part * kSteps + s], C = ZM[part * kSteps + s];
            const float2 X = make_float2(A.x, A.y), Y = make_float2(A.z, A.w);
            const float2 Z = make_float2(C.x, C.y), M = make_float2(C.z, C.w);
            float2 LX, LY, LZ;
            if (kPrecise) {
                const int e = kSym ? (lane + part * kSteps + s) & 31 : part * kSteps + s;
                LX = lx[e];
                LY = ly[e];
                LZ = lz[e];
            }
#pragma unroll
            for (int k = 0; k < I; ++k) {
                float2 dx = __fadd2_rn(X, nx[k]), dy = __fadd2_rn(Y, ny[k]), dz = __fadd2_rn(Z, nz[k]);
                if (kPrecise) {
                    dx = __fadd2_rn(dx, __fadd2_rn(LX, qx[k]));
                    dy = __fadd2_rn(dy, __fadd2_rn(LY, qy[k]));
                    dz = __fadd2_rn(dz, __fadd2_rn(LZ, qz[k]));
                }
                float2 r2 = __fmul2_rn(dx, dx);
                r2 = __ffma2_rn(dy, dy, r2);
                r2 = __ffma2_rn(dz, dz, r2);
                float2 inv = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
                if (kGuard) {
                    inv.x = r2.x > 0.f ? inv.x : 0.f;
                    inv.y = r2.y > 0.f ? inv.y : 0.f;
                }
                const float2 inv2 = __fmul2_rn(inv, inv);
                const float2 sj = __fmul2_rn(__fmul2_rn(M, inv), inv2);
                fx[k] = __ffma2_rn(dx, sj, fx[k]);
                fy[k] = __ffma2_rn(dy, sj, fy[k]);
                fz[k] = __ffma2_rn(dz, sj, fz[k]);
                if (kSym) {
                    const float2 si = __fmul2_rn(__fmul2_rn(mi[k], inv), inv2);
                    cx = __ffma2_rn(dx, si, cx);
                    cy = __ffma2_rn(dy, si, cy);
                    cz = __ffma2_rn(dz, si, cz);
                }
            }
            if (kSym) {
                cx.x = __shfl_sync(0xffffffffu, cx.x, lane + 1);
                cx.y = __shfl_sync(0xffffffffu, cx.y, lane + 1);
                cy.x = __shfl_sync(0xffffffffu, cy.x, lane + 1);
                cy.y = __shfl_sync(0xffffffffu, cy.y, lane + 1);
                cz.x = __shfl_sync(0xffffffffu, cz.x, lane + 1);
                cz.y = __shfl_sync(0xffffffffu, cz.y, lane + 1);
            }
        }
        if (kSym) {  // after S steps and S passes lane l holds packed column (l + S) mod 32
            const int u = (lane + (part + 1) * kSteps) & 31;
            float2 *c = reinterpret_cast<float2 *>(col + part * 3 * tc) + u;
            c[0] = cx;
            c[tc / 2] = cy;
            c[tc] = cz;
        }
    }
}

// Coincident bodies have to be selected away within the aligned runs of kGuarded bodies, as among the rows of
// the widest ordered-pair kernel.  With the close-pair check (kCheck) a warp's threshold is at least FLT_MIN,
// so that a chunk which meets its rows takes the precise path, which guards, also where all its rows lie
// at the centre.  Without the check, an instance of its own guards the tiles of the rows' run: a guarded
// fast path beside the precise one, or zeroed remainders there, cost every caller 2 % (N = 262144).
constexpr int kGuarded = 1024;

template <int I, int T, int TC, int MINB, int U, int NH, int FC, bool kCheck>
__global__ void __launch_bounds__(T, MINB) force_mixed_sym_kernel(SymKArgs a) {
    using Smem = SymMixedSmem<I, T, TC, NH>;
    constexpr int kWarps = Smem::kWarps, kChunks = Smem::kChunks, kFetch = (TC + T - 1) / T;
    static_assert(T % 32 == 0 && TC % 64 == 0, "whole warps and chunks");
    extern __shared__ __align__(16) unsigned char sym_smem[];
    Smem &S = *reinterpret_cast<Smem *>(sym_smem);
    const int t = threadIdx.x, warp = t >> 5;
    const float kInf = __int_as_float(0x7f800000);
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
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
        const int64_t r = S.su[1], c0 = S.su[2], c1 = S.su[3];
        const int64_t row0 = r * a.g.B;
        if (row0 >= a.g.n) {
            __syncthreads();
            continue;
        }
        // the row block's FP32 frame is centred on the mean position of its bodies
        double px[I], py[I], pz[I];
        float2 mi[I];
        double msx = 0.0, msy = 0.0, msz = 0.0;
#pragma unroll
        for (int k = 0; k < I; ++k) {
            const int64_t i = row0 + t * I + k;  // a warp holds 32 I consecutive bodies
            px[k] = py[k] = pz[k] = 0.0;
            float gm = 0.f;
            if (i < a.g.n) {
                const double4 p = a.src[i];
                px[k] = p.x; py[k] = p.y; pz[k] = p.z;
                gm = (float)(a.G * p.w);
                msx += p.x; msy += p.y; msz += p.z;
            }
            mi[k] = make_float2(gm, gm);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            msx += __shfl_xor_sync(0xffffffffu, msx, o);
            msy += __shfl_xor_sync(0xffffffffu, msy, o);
            msz += __shfl_xor_sync(0xffffffffu, msz, o);
        }
        if ((t & 31) == 0) {
            S.cred[0][warp] = msx;
            S.cred[1][warp] = msy;
            S.cred[2][warp] = msz;
        }
        __syncthreads();
        double3 c = make_double3(0.0, 0.0, 0.0);
        for (int w = 0; w < kWarps; ++w) {
            c.x += S.cred[0][w];
            c.y += S.cred[1][w];
            c.z += S.cred[2][w];
        }
        const double inv_rows = 1.0 / (double)min((int64_t)a.g.B, a.g.n - row0);
        c.x *= inv_rows;
        c.y *= inv_rows;
        c.z *= inv_rows;
        float2 nx[I], ny[I], nz[I];
        {
            float blo[3] = {kInf, kInf, kInf}, bhi[3] = {-kInf, -kInf, -kInf}, bth = 0.f;
#pragma unroll
            for (int k = 0; k < I; ++k) {
                const bool real = row0 + t * I + k < a.g.n;  // padding rows sit at the centre, massless
                const double ex = real ? px[k] - c.x : 0.0, ey = real ? py[k] - c.y : 0.0,
                             ez = real ? pz[k] - c.z : 0.0;
                const float x = (float)ex, y = (float)ey, z = (float)ez;
                nx[k] = make_float2(-x, -x);
                ny[k] = make_float2(-y, -y);
                nz[k] = make_float2(-z, -z);
                S.ilo[0][k][t] = (float)(ex - (double)x);
                S.ilo[1][k][t] = (float)(ey - (double)y);
                S.ilo[2][k][t] = (float)(ez - (double)z);
                blo[0] = fminf(blo[0], real ? x : kInf);
                blo[1] = fminf(blo[1], real ? y : kInf);
                blo[2] = fminf(blo[2], real ? z : kInf);
                bhi[0] = fmaxf(bhi[0], real ? x : -kInf);
                bhi[1] = fmaxf(bhi[1], real ? y : -kInf);
                bhi[2] = fmaxf(bhi[2], real ? z : -kInf);
                bth = fmaxf(bth, a.near2 * fmaf(z, z, fmaf(y, y, x * x)));
            }
            const float v0 = warp_minf(blo[0]), v1 = warp_minf(blo[1]), v2 = warp_minf(blo[2]);
            const float v3 = warp_maxf(bhi[0]), v4 = warp_maxf(bhi[1]), v5 = warp_maxf(bhi[2]);
            const float v6 = warp_maxf(bth);
            if ((t & 31) == 0) {
                float *b = S.ibox[warp];
                b[0] = v0; b[1] = v1; b[2] = v2; b[3] = v3; b[4] = v4; b[5] = v5; b[6] = fmaxf(v6, FLT_MIN);
            }
        }
        KahanAcc<I, true, T> acc;
        acc.sm = S.kah;
        acc.init(t);
        // column e of the tile: hi part of x - c, remainder, G m, and the box of each 32 columns
        auto stage = [&](int buf, int e, bool have, const double4 &q) {
            float x = 1e30f, y = 1e30f, z = 1e30f, m = 0.f, l0 = 0.f, l1 = 0.f, l2 = 0.f;  // padding: r2 = inf
            if (have) {
                const double ex = q.x - c.x, ey = q.y - c.y, ez = q.z - c.z;
                x = (float)ex; y = (float)ey; z = (float)ez;
                l0 = (float)(ex - (double)x);
                l1 = (float)(ey - (double)y);
                l2 = (float)(ez - (double)z);
                m = (float)(a.G * q.w);
            }
            const int p = (e >> 6) * 64 + ((e & 63) >> 1), h = e & 1;
            float *A = reinterpret_cast<float *>(S.xy[buf]) + p * 4 + h;
            float *C = reinterpret_cast<float *>(S.zm[buf]) + p * 4 + h;
            A[0] = A[128] = x;
            A[2] = A[130] = y;
            C[0] = C[128] = z;
            C[2] = C[130] = m;
            reinterpret_cast<float *>(S.lx[buf])[e] = l0;
            reinterpret_cast<float *>(S.ly[buf])[e] = l1;
            reinterpret_cast<float *>(S.lz[buf])[e] = l2;
            const float b0 = warp_minf(have ? x : kInf), b1 = warp_minf(have ? y : kInf);
            const float b2 = warp_minf(have ? z : kInf), b3 = warp_maxf(have ? x : -kInf);
            const float b4 = warp_maxf(have ? y : -kInf), b5 = warp_maxf(have ? z : -kInf);
            if ((e & 31) == 0) {
                float *b = S.jbox[buf][e >> 5];
                b[0] = b0; b[1] = b1; b[2] = b2; b[3] = b3; b[4] = b4; b[5] = b5;
            }
        };
        const int64_t own_end = (r / a.g.s + 1) * a.g.kw;
        const int64_t coff = sym_col_off(a.g, r) - a.col0 - own_end;
        if (c0 < c1) {
            for (int e = t; e < TC; e += T) {  // whole warps stage together
                const int64_t j = c0 * TC + e;
                const bool have = j < a.g.n;
                stage(0, e, have, have ? a.src[j] : make_double4(0.0, 0.0, 0.0, 0.0));
            }
        }
        __syncthreads();
        int cur = 0;
        const float *iw = S.ibox[warp];
        for (int64_t jt = c0; jt < c1; ++jt, cur ^= 1) {
            const bool more = jt + 1 < c1, sym = jt >= own_end;
            double4 qn[kFetch];
#pragma unroll
            for (int f = 0; f < kFetch; ++f) {
                const int64_t j = (jt + 1) * TC + t + f * T;
                qn[f] = more && t + f * T < TC && j < a.g.n ? a.src[j] : make_double4(0.0, 0.0, 0.0, 0.0);
            }
            float2 fx[I], fy[I], fz[I];
#pragma unroll
            for (int k = 0; k < I; ++k) fx[k] = fy[k] = fz[k] = make_float2(0.f, 0.f);
#pragma unroll 1
            for (int ch = 0; ch < kChunks; ++ch) {
                // smallest possible squared distance between the warp's rows and the chunk's columns
                const float(*cb)[6] = &S.jbox[cur][ch * 2];
                float g2 = 0.f;
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const float lo = fminf(cb[0][d], cb[1][d]), hi = fmaxf(cb[0][3 + d], cb[1][3 + d]);
                    const float g = fmaxf(0.f, fmaxf(lo - iw[3 + d], iw[d] - hi));
                    g2 = fmaf(g, g, g2);
                }
                const bool precise = kCheck && g2 < iw[6];
                const float4 *xy = S.xy[cur] + ch * 64, *zm = S.zm[cur] + ch * 64;
                const float2 *lx = S.lx[cur] + ch * 32, *ly = S.ly[cur] + ch * 32, *lz = S.lz[cur] + ch * 32;
                float *col = &S.col[cur][warp][0][0][ch * 64];
                if (sym) {
                    if (precise)
                        sym_mixed_chunk<I, T, 2, NH, true, true>(xy, zm, lx, ly, lz, S.ilo, nx, ny, nz, mi, fx, fy, fz, col, TC);
                    else if (!kCheck && jt < (row0 / kGuarded + 1) * (kGuarded / TC))
                        sym_mixed_chunk<I, T, 2, NH, true, false, true>(xy, zm, lx, ly, lz, S.ilo, nx, ny, nz, mi, fx, fy, fz, col, TC);
                    else
                        sym_mixed_chunk<I, T, U, NH, true, false>(xy, zm, lx, ly, lz, S.ilo, nx, ny, nz, mi, fx, fy, fz, col, TC);
                } else {
                    if (precise)
                        sym_mixed_chunk<I, T, 1, NH, false, true>(xy, zm, lx, ly, lz, S.ilo, nx, ny, nz, mi, fx, fy, fz, col, TC);
                    else
                        sym_mixed_chunk<I, T, 2, NH, false, false>(xy, zm, lx, ly, lz, S.ilo, nx, ny, nz, mi, fx, fy, fz, col, TC);
                }
                if (FC == 64 || (ch & 1) || ch + 1 == kChunks) {
#pragma unroll
                    for (int k = 0; k < I; ++k) {
                        acc.add(0, k, (double)fx[k].x + (double)fx[k].y);
                        acc.add(1, k, (double)fy[k].x + (double)fy[k].y);
                        acc.add(2, k, (double)fz[k].x + (double)fz[k].y);
                        fx[k] = fy[k] = fz[k] = make_float2(0.f, 0.f);
                    }
                }
            }
            if (more) {
#pragma unroll
                for (int f = 0; f < kFetch; ++f) {
                    const int e = t + f * T;
                    if (e < TC) stage(cur ^ 1, e, (jt + 1) * TC + e < a.g.n, qn[f]);
                }
            }
            __syncthreads();
            if (sym) {
                double *slot = a.colpart + (size_t)(coff + jt) * 3 * TC;
                const float *cs = &S.col[cur][0][0][0][0];
#pragma unroll
                for (int e = t; e < 3 * TC; e += T)
                    slot[e] = -sym_tree<kWarps * NH>([&](int w) { return (double)cs[w * 3 * TC + e]; });
            }
        }
        double *slot = a.rowpart + (size_t)(u - a.unit0) * 3 * a.g.B;
#pragma unroll
        for (int k = 0; k < I; ++k) {
            const int l = t * I + k;
            slot[l] = acc.result(0, k);
            slot[a.g.B + l] = acc.result(1, k);
            slot[2 * a.g.B + l] = acc.result(2, k);
        }
        __syncthreads();
    }
}

// -------------------------------------------------------------------------------------------
// The sum of a body's row and column slots
// -------------------------------------------------------------------------------------------
struct SymReduceArgs {
    SymSlots slots;
    double *out3;  // mode 0: the running sum to write (3 arrays of n); mode 2: triples
    int mode;      // 0 running sum, 1 epilogue, 2 triples
    StepArgs st;
    int epi;
    unsigned *queue;  // the batch's counter, for the next evaluation
};

__global__ void __launch_bounds__(kRedWarps * 32) sym_reduce_kernel(SymReduceArgs a) {
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.queue = 0;
    sym_reduce<3>(a.slots, [&](int64_t i, const double (&v)[3]) {
        if (a.mode == 1) {
            apply_epilogue(a.st, a.epi, i, v[0], v[1], v[2]);
        } else if (a.mode == 0) {
#pragma unroll
            for (int d = 0; d < 3; ++d) a.out3[(size_t)d * a.slots.g.n + i] = v[d];
        } else {
#pragma unroll
            for (int d = 0; d < 3; ++d) a.out3[3 * i + d] = v[d];
        }
    });
}

// -------------------------------------------------------------------------------------------
// Plan and launch
// -------------------------------------------------------------------------------------------
// FP64: 0 up to N = 32768, 1 above (the wider group selects coincident bodies away over the same 1024
// bodies as the ordered kernel that ran there).  Mixed: 0 folds a row after 128 columns and a column
// after 16 steps (64 terms per packed half), as the ordered kernel does from N = 32768; 1 folds both
// twice as often, as it does below.  A unit's own cost is higher in the mixed kernel (its rows' frame and
// boxes); with the FP64 kernel's 0.1 the units came out too short: N = 12000 116 us a step against 104,
// 40000 672 against 650.
static const SymShape kSymF64[] = {{4, 128, 64, 512}, {4, 128, 128, 1024}};
static const SymShape kSymMixed[] = {{4, 128, 128, 512, 0.3}, {4, 128, 64, 512, 0.3}};

SymShape sym_shape(int precision, int kind) { return precision == GTD_PREC_MIXED ? kSymMixed[kind] : kSymF64[kind]; }

template <typename F>
static void with_sym(int precision, int kind, bool check, F &&f) {
    if (precision == GTD_PREC_MIXED) {
        constexpr size_t s1 = sizeof(SymMixedSmem<4, 128, 64, 4>), s0 = sizeof(SymMixedSmem<4, 128, 128, 2>);
        if (kind == 1 && check) f(force_mixed_sym_kernel<4, 128, 64, 3, 8, 4, 64, true>, s1);
        else if (kind == 1) f(force_mixed_sym_kernel<4, 128, 64, 3, 8, 4, 64, false>, s1);
        else if (check) f(force_mixed_sym_kernel<4, 128, 128, 3, 4, 2, 128, true>, s0);
        else f(force_mixed_sym_kernel<4, 128, 128, 3, 4, 2, 128, false>, s0);
    } else {
        if (kind == 1) f(force_f64_sym_kernel<4, 128, 128, 3>, (size_t)0);
        else f(force_f64_sym_kernel<4, 128, 64, 3>, (size_t)0);
    }
}

size_t sym_partial_bytes(const ForcePlan &p) { return sym_layout(p.sg, p.sym_bytes, 3).bytes; }

int sym_make_plan(ForcePlan &p, int precision, int kind, int sms) {
    const SymShape sh = sym_shape(precision, kind);
    int per_sm = 1;
    with_sym(precision, kind, true, [&](auto k, size_t smem) {
        if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, sh.threads, smem);
    });
    if (per_sm < 1) per_sm = 1;
    const int64_t ctas = (int64_t)sms * per_sm;
    const SymGeom g = sym_geometry(p.n, sh, sms, per_sm);
    p.sym = true;
    p.sym_kind = kind;
    p.sg = g;
    p.bi = g.B;
    p.bj = g.TC;
    p.rows = (p.n + g.B - 1) / g.B;
    p.tiles = g.nt;
    p.total = p.rows * p.tiles;
    p.units = sym_tri(g, g.Gs) * sym_block_units(g);
    p.grid = (int)std::min<int64_t>(ctas, p.units);
    return GTD_OK;
}

// Shrinks the plan's partial sums to at most max_bytes (more and smaller batches); GTD_ERR_CAPACITY where
// even one super-group a batch does not fit.
int sym_fit(ForcePlan &p, size_t max_bytes) {
    SymGeom &g = p.sg;
    // fewer row slots where that saves a batch and leaves some units per CTA
    while (g.q == 1 && sym_slot_bytes(g, 0, g.Gs) > max_bytes && p.units / 2 >= 6 * (int64_t)p.grid) {
        g.L *= 2;
        g.Gs = (g.G + g.L - 1) / g.L;
        p.units = sym_tri(g, g.Gs) * sym_block_units(g);
    }
    // the slots get what the counters and the running sum leave
    const size_t fixed = (size_t)3 * p.n * sizeof(double) + 512 + (size_t)g.Gs * sizeof(unsigned);
    p.sym_bytes = max_bytes > fixed ? max_bytes - fixed : 0;
    if (sym_partial_bytes(p) > max_bytes)
        return fail(GTD_ERR_CAPACITY, "%lld bodies need more partial sums than %zu bytes hold", (long long)p.n, max_bytes);
    return GTD_OK;
}

int sym_reset(const ForcePlan &p, double *partials, cudaStream_t s) {
    GTD_CUDA(cudaMemsetAsync(partials, 0, (size_t)sym_layout(p.sg, p.sym_bytes, 3).batches * sizeof(unsigned), s));
    return GTD_OK;
}

// The force kernels and reductions of a handle's steps are chained launches.  A KDK step with the counter
// cleared each time and full launches, and so, us: FP64 5000 37.2 / 35.1, 16384 220 / 215; mixed 5000
// 40.8 / 36.9, 16384 166 / 160.
int sym_launch_force(int precision, const ForcePlan &p, const double4 *src, double G, double *partials, bool chained,
                     cudaStream_t s) {
    const SymGeom &g = p.sg;
    const SymLayout lay = sym_layout(g, p.sym_bytes, 3);
    char *mem = reinterpret_cast<char *>(partials);
    int64_t batch = 0;
    for (int64_t Pa = 0; Pa < g.Gs; ++batch) {
        const int64_t Pb = sym_batch_end(g, Pa, p.sym_bytes);
        SymReduceArgs r{};
        r.slots = sym_slots(g, lay, mem, Pa, Pb, 3);
        SymKArgs a{};
        a.g = g;
        a.src = src;
        a.G = G;
        a.rowpart = const_cast<double *>(r.slots.rowpart);
        a.colpart = const_cast<double *>(r.slots.colpart);
        a.unit0 = r.slots.unit0;
        a.unit1 = sym_tri(g, Pb) * sym_block_units(g);
        a.col0 = r.slots.col0;
        a.near2 = p.near2;
        a.queue = reinterpret_cast<unsigned *>(mem) + batch;
        const int grid = (int)std::min<int64_t>(p.grid, a.unit1 - a.unit0);
        cudaError_t e = cudaSuccess;
        with_sym(precision, p.sym_kind, p.near2 > 0.f, [&](auto k, size_t smem) {
            if (smem > 48 * 1024) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e == cudaSuccess) launch_chained(chained, k, grid, sym_shape(precision, p.sym_kind).threads, smem, s, a);
        });
        GTD_CUDA(e);
        GTD_CHECK_LAUNCH();
        if (Pb < g.Gs) {
            r.mode = 0;
            r.out3 = reinterpret_cast<double *>(mem + lay.base);
            r.queue = a.queue;
            launch_chained(chained, sym_reduce_kernel, (unsigned)((g.n + 31) / 32), kRedWarps * 32, 0, s, r);
            GTD_CHECK_LAUNCH();
        }
        Pa = Pb;
    }
    return GTD_OK;
}

int sym_launches(const ForcePlan &p) { return 2 * (int)sym_layout(p.sg, p.sym_bytes, 3).batches; }

// The last batch's sums, with the earlier ones', into the epilogue (acc3 == NULL) or acc3.
int sym_launch_finish(const ForcePlan &p, const double *partials, int epi, const StepArgs &st, double *acc3, bool chained,
                      cudaStream_t s) {
    const SymGeom &g = p.sg;
    const SymLayout lay = sym_layout(g, p.sym_bytes, 3);
    int64_t Pa = 0, Pb = sym_batch_end(g, 0, p.sym_bytes);
    for (; Pb < g.Gs; Pb = sym_batch_end(g, Pa, p.sym_bytes)) Pa = Pb;
    SymReduceArgs r{};
    r.queue = const_cast<unsigned *>(reinterpret_cast<const unsigned *>(partials)) + lay.batches - 1;
    r.slots = sym_slots(g, lay, reinterpret_cast<const char *>(partials), Pa, Pb, 3);
    r.mode = acc3 ? 2 : 1;
    r.out3 = acc3;
    r.st = st;
    r.epi = epi;
    launch_chained(chained, sym_reduce_kernel, (unsigned)((g.n + 31) / 32), kRedWarps * 32, 0, s, r);
    GTD_CHECK_LAUNCH();
    return GTD_OK;
}

}  // namespace gtd

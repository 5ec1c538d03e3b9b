// Batched ensemble of independent few-body systems: one persistent launch advances every system
// by one leapfrog KDK step (gregsys.hpp:2946-2990 per system), the step loop is captured in a CUDA
// graph, and overlap merges (body::operator+=, the check_overlap scan) run inside the same launch.
//
// This is the device form of the reference drivers' ensemble pattern - one gtd::system per
// std::thread (bdsim.cpp:82-113) - with FP64 state and FP32 pair forces.
//
// Work decomposition: a CTA takes one item, a chunk of IB rows per thread of one system, and the items
// start largest system first, so the spread in per-system work (N = 3 .. 2048: 4.7e5x in pairs) balances
// across the GPU; with a CTA per system the largest alone set the step time (512 systems of up to 2048
// bodies: 0.60 ms a step, 0.38 with items).  The CTA that finishes a system's last chunk (a count of
// arrivals, no waiting) also takes its merges and the next step's kick and drift, so a step stays one
// launch.  Each CTA stages the whole system in shared memory as FP32 coordinates relative to the
// system's mean position, with G m; its rows are spread over the threads, IB (1, 2 or 4) each,
// and each thread sums its rows' forces two j-bodies per packed FP32x2 instruction, folding every
// 64 j-bodies into FP64.  Alongside the force it keeps the smallest separation to any other body (a
// 3-input float minimum; in the one fold holding the row's own body its j pair is left out by number, not
// by its value, which coincident bodies share); a body closer to another than its radius plus the system's
// largest radius, plus a bound on the FP32 staging error, flags the row; only systems with flagged rows run
// the exact FP64 merge scan, over those rows.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <new>
#include <numeric>
#include <vector>

#include "ensemble_rows.cuh"
#include "gtd_internal.cuh"
#include "host_copy.cuh"

namespace gtd {
struct EnsCand;
struct EnsInfo;
}

struct gtd_ensemble {
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    double G = 6.6743e-11, dt = 1.0;
    int merge = 1;
    int threads = 256;   // CTA size
    int ib = 1;          // bodies per thread in the force loop (2 and 4 need threads <= 256)
    bool configured = false;  // both set by the caller or the autotuner; else ens_default chooses at upload
    int64_t n_sys = 0, n_bodies = 0;
    int max_n = 0;
    std::vector<int64_t> off_h;       // [n_sys+1]
    std::vector<int32_t> order_h;     // systems, largest first
    int64_t *off = nullptr;           // [n_sys+1]
    int32_t *cnt = nullptr;           // live bodies per system
    int32_t *order = nullptr;         // systems, largest first
    double4 *pos = nullptr, *vel = nullptr, *acc = nullptr;
    double *rad = nullptr, *rest = nullptr;
    int32_t *ids = nullptr;
    unsigned *merged = nullptr;       // merges so far
    gtd::EnsCand *cand = nullptr;     // [n_sys] rows the separation test flagged
    gtd::EnsInfo *info = nullptr;     // [n_sys] frame of the staged coordinates
    int *arrived = nullptr;           // [n_sys] chunks finished in this launch
    int2 *items = nullptr;            // (system, first row), largest system first
    int64_t n_items = 0;
    int items_for = 0;                // the (threads, ib) the items were made for
    double *io = nullptr;             // host arrays on the device: x3 | v3 | a3 | m | r | rest
    gtd::HostRing host_ring;
    bool begun = false;
    uint64_t launches = 0;
    cudaGraphExec_t graph = nullptr;
    int graph_steps = 0;
    int graph_threads = 0;
};

namespace gtd {

constexpr int kEnsMaxN = 8192;
constexpr int kEnsFold = 64;

constexpr int kEnsCand = 256;  // candidate rows a system's scan tracks before it falls back to the full scan

struct EnsCand {
    int n;                 // candidates listed (may exceed kEnsCand: then the list is incomplete)
    int o, num, next;      // scan state: current row, rows, the partner found (-1: none, -2: done)
    int restarted;
    int row[kEnsCand];
};

// Frame of a system's staged coordinates and what its separation test needs.
struct EnsInfo {
    double cx, cy, cz;  // mean position
    float rmax, floor2, slack;
};

struct EnsArgs {
    const int64_t *off;
    int32_t *cnt;
    const int32_t *order;  // systems, largest first
    const int2 *items;
    double4 *pos, *vel, *acc;
    double *rad, *rest;
    int32_t *ids;
    EnsCand *cand;
    EnsInfo *info;
    int *arrived;
    double G, h;
    int kick;    // close the step with a half kick (0: the initial force)
    int pre;     // then open the next one: half kick and drift
    int merge;
    int chunk;   // rows per item
    int stride;  // floats per staged coordinate array (largest system, rounded up to even)
    unsigned *merged;
};

__device__ __forceinline__ float ens_rsqrt(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Smallest r2 floor that keeps the self pair's G m / r^3 finite in FP32 for every body of a system
// whose largest G m is Gm: floor^(3/2) >= Gm * 2^-120, and at least 2^-100 (a normal float whose
// 1/r^2 = 2^100 stays finite).  For G m = 6.7e20 (1e31 kg, SI) that is 6.3e-11 m^2: it changes r2
// only for pairs closer than ~5 cm, far inside the FP32 resolution of the staged coordinates.
__device__ __forceinline__ float ens_r2_floor(float Gm) {
    const double c = cbrt((double)Gm * 0x1p-120);
    const double f = c * c;
    return f > 0x1p-100 ? (float)f : 0x1p-100f;
}

__device__ void ens_merge_into(double4 &po, double4 &vo, double4 &ao, double &ro, double &eo, const double4 &pi,
                               const double4 &vi, const double4 &ai, double ri, double ei) {
    const double ma = po.w, mb = pi.w, ms = __dadd_rn(ma, mb);
    auto mix = [&](double a, double b) { return __ddiv_rn(__dadd_rn(__dmul_rn(ma, a), __dmul_rn(mb, b)), ms); };
    const double4 np = make_double4(mix(po.x, pi.x), mix(po.y, pi.y), mix(po.z, pi.z), ms);
    const double4 nv = make_double4(mix(vo.x, vi.x), mix(vo.y, vi.y), mix(vo.z, vi.z), 0.0);
    const double4 na = make_double4(mix(ao.x, ai.x), mix(ao.y, ai.y), mix(ao.z, ai.z), 0.0);
    eo = 0.5 * (eo + ei);
    ro = cbrt(__dadd_rn(__dmul_rn(__dmul_rn(ro, ro), ro), __dmul_rn(__dmul_rn(ri, ri), ri)));
    po = np;
    vo = nv;
    ao = na;
}

__device__ __forceinline__ bool ens_overlaps(const double4 &a, double ra, const double4 &b, double rb) {
    const double dx = __dsub_rn(b.x, a.x), dy = __dsub_rn(b.y, a.y), dz = __dsub_rn(b.z, a.z);
    const double d = sqrt(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
    return d < __dadd_rn(ra, rb);
}

// Removes row i of a system of num rows (the vector erase of the reference's scan): rows i+1 .. num-1
// move down by one, in passes of T rows.
__device__ __noinline__ void ens_erase_row(int i, int num, double4 *pos, double4 *vel, double4 *acc, double *rad, double *rest,
                              int32_t *ids) {
    const int t = threadIdx.x, T = blockDim.x;
    for (int base = i; base < num - 1; base += T) {
        const int k = base + t;
        const bool act = k < num - 1;
        double4 p, v, a;
        double r = 0, e = 0;
        int32_t id = 0;
        if (act) { p = pos[k + 1]; v = vel[k + 1]; a = acc[k + 1]; r = rad[k + 1]; e = rest[k + 1]; id = ids[k + 1]; }
        __syncthreads();
        if (act) { pos[k] = p; vel[k] = v; acc[k] = a; rad[k] = r; rest[k] = e; ids[k] = id; }
        __syncthreads();
    }
}

// The check_overlap scan (merges, restart from index 0 after each) over one system, by one CTA,
// from scan state (n rows, at row o0, restarted0: the last step merged into o0).
__device__ __noinline__ int ens_merge_scan(int n, int o0, bool restarted0, double4 *pos, double4 *vel, double4 *acc, double *rad,
                              double *rest, int32_t *ids, int *sh) {
    // sh[0] = best, sh[1] = num, sh[2] = o
    const int t = threadIdx.x, T = blockDim.x;
    if (t == 0) {
        sh[1] = n;
        sh[2] = o0;
    }
    __syncthreads();
    bool restarted = restarted0;
    while (true) {
        const int num = sh[1], o = sh[2];
        if (o >= num) break;
        const int lo = restarted ? 0 : o + 1;
        if (t == 0) sh[0] = INT32_MAX;
        __syncthreads();
        const double4 po = pos[o];
        const double ro = rad[o];
        for (int i = lo + t; i < num; i += T)
            if (i != o && ens_overlaps(po, ro, pos[i], rad[i])) atomicMin(&sh[0], i);
        __syncthreads();
        const int i = sh[0];
        if (i == INT32_MAX) {
            if (t == 0) sh[2] = o + 1;
            restarted = false;
            __syncthreads();
            continue;
        }
        if (t == 0) {
            double4 p = pos[o], v = vel[o], a = acc[o];
            double r = rad[o], e = rest[o];
            ens_merge_into(p, v, a, r, e, pos[i], vel[i], acc[i], rad[i], rest[i]);
            pos[o] = p; vel[o] = v; acc[o] = a; rad[o] = r; rest[o] = e;
        }
        __syncthreads();
        ens_erase_row(i, num, pos, vel, acc, rad, rest, ids);
        if (t == 0) {
            sh[1] = num - 1;
            sh[2] = i < o ? o - 1 : o;
        }
        restarted = true;
        __syncthreads();
    }
    const int out = sh[1];
    __syncthreads();
    return out;
}

// One step of the candidate scan, by one thread: sorts and de-duplicates the list, finds the next
// (row, partner) pair in scan order from the state in c and merges the partner into the row
// (c.next = the partner), or ends the scan (c.next = -2).
__device__ __noinline__ void ens_cand_next(double4 *pos, double4 *vel, double4 *acc, double *rad, double *rest,
                                           EnsCand &c) {
    // sort the list (few entries; insertion sort) and drop duplicates
    int k = 0;
    for (int a = 0; a < c.n; ++a) {
        const int v = c.row[a];
        int b = k;
        while (b > 0 && c.row[b - 1] > v) { c.row[b] = c.row[b - 1]; --b; }
        c.row[b] = v;
        ++k;
    }
    int u = 0;
    for (int a = 0; a < k; ++a)
        if (u == 0 || c.row[u - 1] != c.row[a]) c.row[u++] = c.row[a];
    c.n = u;
    int o = c.o;
    bool restarted = c.restarted != 0;
    int found = -2;
    while (true) {
        if (!restarted) {  // jump to the first candidate at or after o
            int a = 0;
            while (a < c.n && c.row[a] < o) ++a;
            if (a == c.n) break;
            o = c.row[a];
        }
        const int lo = restarted ? 0 : o + 1;
        const double4 po = pos[o];
        const double ro = rad[o];
        int best = -1;
        for (int a = 0; a < c.n; ++a) {
            const int i = c.row[a];
            if (i >= lo && i != o && ens_overlaps(po, ro, pos[i], rad[i])) {
                best = i;  // the list is sorted: the first partner is the smallest
                break;
            }
        }
        if (best >= 0) {
            found = best;
            break;
        }
        ++o;
        restarted = false;
    }
    c.o = o;
    c.next = found;
    if (found >= 0) {
        double4 p = pos[o], v = vel[o], a = acc[o];
        double r = rad[o], e = rest[o];
        ens_merge_into(p, v, a, r, e, pos[found], vel[found], acc[found], rad[found], rest[found]);
        pos[o] = p; vel[o] = v; acc[o] = a; rad[o] = r; rest[o] = e;
    }
}

// The same scan restricted to candidate rows.  Every row with an FP64 overlap partner was flagged
// by the force loop's FP32 separation test (a bound that covers the staging error), and overlap is
// symmetric, so a row outside the list overlaps nothing and its partners are all listed: the scan
// can jump from candidate to candidate and search the list alone, taking the same merges in the same
// order as the full scan.  After a merge only the merged row has moved; it is tested against every
// row and its new partners join the list.  Returns the rows left; if the list overflows, the full
// scan continues from the state reached.
__device__ __noinline__ int ens_merge_scan_cand(int n, double4 *pos, double4 *vel, double4 *acc, double *rad, double *rest,
                                   int32_t *ids, EnsCand &c, int *sh) {
    const int t = threadIdx.x;
    if (t == 0) {
        c.o = 0;
        c.num = n;
        c.restarted = 0;
    }
    while (true) {
        if (t == 0) ens_cand_next(pos, vel, acc, rad, rest, c);
        __syncthreads();
        const int i = c.next, num = c.num;
        __syncthreads();  // every thread has read the state before thread 0 changes it
        if (i < 0) break;
        ens_erase_row(i, num, pos, vel, acc, rad, rest, ids);
        if (t == 0) {
            // the list after the erase: i leaves, later rows move down by one
            int u = 0;
            for (int a = 0; a < c.n; ++a) {
                const int r = c.row[a];
                if (r != i) c.row[u++] = r > i ? r - 1 : r;
            }
            c.n = u;
            c.o = i < c.o ? c.o - 1 : c.o;
            c.num = num - 1;
            c.restarted = 1;
        }
        __syncthreads();
        // the merged row's partners join the list (with the merged row itself)
        const int o = c.o, nm = c.num;
        const double4 po = pos[o];
        const double ro = rad[o];
        bool any = false;
        for (int k = t; k < nm; k += blockDim.x)
            if (k != o && ens_overlaps(po, ro, pos[k], rad[k])) {
                const int s = atomicAdd(&c.n, 1);
                if (s < kEnsCand) c.row[s] = k;
                any = true;
            }
        if (__syncthreads_or(any) && t == 0) {
            const int s = atomicAdd(&c.n, 1);
            if (s < kEnsCand) c.row[s] = o;
        }
        __syncthreads();
        const bool overflow = c.n > kEnsCand;
        const int o1 = c.o, n1 = c.num;
        __syncthreads();
        if (overflow)  // too many to track: the full scan from here
            return ens_merge_scan(n1, o1, true, pos, vel, acc, rad, rest, ids, sh);
    }
    const int out = c.num;
    __syncthreads();
    return out;
}

__device__ __forceinline__ float ens_min3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// One fold (j pairs q0 .. q1-1) of the force loop for IB rows, with the smallest r2 to another body.  kOwn:
// the fold holds one of the rows' own bodies, whose j pair oq[b] stays out of the minimum (its other body is
// in it from the start).  Leaving out a vanishing r2 instead leaves out coincident bodies too; us a step so and
// by number: 4096 systems of up to 64 bodies 52.4 / 52.9, 256 123.5 / 125.2, 512 of 2048 604 / 612, 64 of 8192
// 1551 / 1492.
template <int IB, bool kOwn>
__device__ __forceinline__ void ens_fold(int q0, int q1, const float2 *X2, const float2 *Y2, const float2 *Z2,
                                         const float2 *M2, const float2 (&nx)[IB], const float2 (&ny)[IB],
                                         const float2 (&nz)[IB], float2 fl2, const int (&oq)[IB],
                                         float2 (&fx)[IB], float2 (&fy)[IB], float2 (&fz)[IB], float (&mn)[IB]) {
#pragma unroll 4
    for (int q = q0; q < q1; ++q) {
        const float2 X = X2[q], Y = Y2[q], Z = Z2[q], M = M2[q];
#pragma unroll
        for (int b = 0; b < IB; ++b) {
            const float2 dx = __fadd2_rn(X, nx[b]), dy = __fadd2_rn(Y, ny[b]), dz = __fadd2_rn(Z, nz[b]);
            float2 r2 = __ffma2_rn(dx, dx, fl2);
            r2 = __ffma2_rn(dy, dy, r2);
            r2 = __ffma2_rn(dz, dz, r2);
            if (!kOwn || q != oq[b]) mn[b] = ens_min3(mn[b], r2.x, r2.y);
            const float2 inv = make_float2(ens_rsqrt(r2.x), ens_rsqrt(r2.y));
            const float2 inv2 = __fmul2_rn(inv, inv);
            float2 sc = __fmul2_rn(M, inv);
            sc = __fmul2_rn(sc, inv2);
            fx[b] = __ffma2_rn(dx, sc, fx[b]);
            fy[b] = __ffma2_rn(dy, sc, fy[b]);
            fz[b] = __ffma2_rn(dz, sc, fz[b]);
        }
    }
}

// Forces on the IB rows r0, r0 + s, ..., r0 + (IB-1) s (those below nc) of a staged system: each
// staged j pair is read from shared memory once for all IB rows.  Returns whether any of them may
// overlap another body.  floor2 is added to every r2 inside its first FMA (no extra instruction):
// the self pair gets r2 = floor2 exactly, a finite 1/r and a zero term (dx = 0).  floor2 is far
// below the staged coordinates' resolution (ens_r2_floor).  r0 - t and s are multiples of 32, so
// the 32 rows of a warp share one fold of kEnsFold j-bodies for each b, and the choice of fold form
// (ens_fold's kOwn) is uniform across the warp.
template <int IB>
__device__ __forceinline__ int ens_force_rows(int r0, int s, int nc, int npad, const float *sx, const float *sy,
                                              const float *sz, const float *sm, double4 *pos, double4 *vel,
                                              double4 *acc, const double *rad, float rmx, float slack, bool kick,
                                              double h2, float floor2, EnsCand *cand) {
    const float2 *X2 = reinterpret_cast<const float2 *>(sx);
    const float2 *Y2 = reinterpret_cast<const float2 *>(sy);
    const float2 *Z2 = reinterpret_cast<const float2 *>(sz);
    const float2 *M2 = reinterpret_cast<const float2 *>(sm);
    float2 nx[IB], ny[IB], nz[IB];
    double ax[IB], ay[IB], az[IB];
    float mn[IB];             // smallest r2 to another body
    int own[IB];              // fold of the row's own body
    int oq[IB];               // its j pair
#pragma unroll
    for (int b = 0; b < IB; ++b) {
        const int ic = ens_staged_row(r0 + b * s, r0, nc);
        nx[b] = make_float2(-sx[ic], -sx[ic]);
        ny[b] = make_float2(-sy[ic], -sy[ic]);
        nz[b] = make_float2(-sz[ic], -sz[ic]);
        ax[b] = ay[b] = az[b] = 0.0;
        const float dx = sx[ic ^ 1] + nx[b].x, dy = sy[ic ^ 1] + ny[b].x, dz = sz[ic ^ 1] + nz[b].x;
        mn[b] = fmaf(dz, dz, fmaf(dy, dy, fmaf(dx, dx, floor2)));  // padding: infinite
        oq[b] = ic >> 1;
        own[b] = ens_stand_in(r0 + b * s, r0, nc) / kEnsFold;
    }
    const float2 fl2 = make_float2(floor2, floor2);
    for (int q0 = 0; q0 < npad / 2; q0 += kEnsFold / 2) {
        const int q1 = min(q0 + kEnsFold / 2, npad / 2);
        const int fold = q0 / (kEnsFold / 2);
        float2 fx[IB], fy[IB], fz[IB];
#pragma unroll
        for (int b = 0; b < IB; ++b) fx[b] = fy[b] = fz[b] = make_float2(0.f, 0.f);
        bool mine = false;
#pragma unroll
        for (int b = 0; b < IB; ++b) mine |= own[b] == fold;
        if (__any_sync(0xffffffffu, mine))
            ens_fold<IB, true>(q0, q1, X2, Y2, Z2, M2, nx, ny, nz, fl2, oq, fx, fy, fz, mn);
        else
            ens_fold<IB, false>(q0, q1, X2, Y2, Z2, M2, nx, ny, nz, fl2, oq, fx, fy, fz, mn);
#pragma unroll
        for (int b = 0; b < IB; ++b) {
            ax[b] += (double)fx[b].x + (double)fx[b].y;
            ay[b] += (double)fy[b].x + (double)fy[b].y;
            az[b] += (double)fz[b].x + (double)fz[b].y;
        }
    }
    int flagged = 0;
#pragma unroll
    for (int b = 0; b < IB; ++b) {
        const int i = r0 + b * s;
        if (i >= nc) continue;
        const float mind2 = mn[b];
        if (mind2 < INFINITY) {  // some other body exists
            const float reach = ((float)rad[i] + rmx) * 1.00001f + slack;
            if (mind2 < reach * reach * 1.0001f + floor2) {
                flagged = 1;
                if (cand) {
                    const int k = atomicAdd(&cand->n, 1);
                    if (k < kEnsCand) cand->row[k] = i;
                }
            }
        }
        if (kick) {
            double4 v = vel[i];
            v.x = fma(h2, ax[b], v.x); v.y = fma(h2, ay[b], v.y); v.z = fma(h2, az[b], v.z);
            vel[i] = v;
        }
        acc[i] = make_double4(ax[b], ay[b], az[b], 0.0);
    }
    return flagged;
}

__device__ __forceinline__ double4 ens_ldcg(const double4 *p) {  // past the L1: another CTA may have written it
    const double2 a = __ldcg(reinterpret_cast<const double2 *>(p)), b = __ldcg(reinterpret_cast<const double2 *>(p) + 1);
    return make_double4(a.x, a.y, b.x, b.y);
}

// Half kick and drift of a system's n rows (with pre), then its frame, by one CTA.  The frame is left in
// shared memory (o) and in *out.
struct EnsBeginSmem {
    double red[3][32];
    float redr[32], redg[32];
    EnsInfo o;
    int xmax_bits;  // largest staged |coordinate| (non-negative float bits)
};
__device__ __noinline__ void ens_begin(int n, double G, double h, int pre, double4 *pos, double4 *vel, const double4 *acc,
                                       const double *rad, EnsInfo *out, EnsBeginSmem &S) {
    const int t = threadIdx.x, T = blockDim.x, lane = t & 31, warp = t >> 5, nw = (T + 31) >> 5;
    const double h2 = 0.5 * h;
    double cx = 0.0, cy = 0.0, cz = 0.0;
    float rmax = 0.f, gmax = 0.f;
    for (int i = t; i < n; i += T) {
        double4 p = ens_ldcg(&pos[i]);
        if (pre) {
            double4 v = ens_ldcg(&vel[i]);
            const double4 ac = ens_ldcg(&acc[i]);
            v.x = fma(h2, ac.x, v.x); v.y = fma(h2, ac.y, v.y); v.z = fma(h2, ac.z, v.z);
            p.x = fma(h, v.x, p.x); p.y = fma(h, v.y, p.y); p.z = fma(h, v.z, p.z);
            vel[i] = v;
            pos[i] = p;
        }
        cx += p.x; cy += p.y; cz += p.z;
        rmax = fmaxf(rmax, (float)__ldcg(&rad[i]));
        gmax = fmaxf(gmax, (float)(G * p.w));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        cx += __shfl_xor_sync(0xffffffffu, cx, o);
        cy += __shfl_xor_sync(0xffffffffu, cy, o);
        cz += __shfl_xor_sync(0xffffffffu, cz, o);
        rmax = fmaxf(rmax, __shfl_xor_sync(0xffffffffu, rmax, o));
        gmax = fmaxf(gmax, __shfl_xor_sync(0xffffffffu, gmax, o));
    }
    if (lane == 0) {
        S.red[0][warp] = cx; S.red[1][warp] = cy; S.red[2][warp] = cz;
        S.redr[warp] = rmax;
        S.redg[warp] = gmax;
    }
    __syncthreads();
    if (t == 0) {
        double X = 0, Y = 0, Z = 0;
        float R = 0.f, Gm = 0.f;
        for (int w = 0; w < nw; ++w) {
            X += S.red[0][w]; Y += S.red[1][w]; Z += S.red[2][w];
            R = fmaxf(R, S.redr[w]);
            Gm = fmaxf(Gm, S.redg[w]);
        }
        S.o.cx = X / n; S.o.cy = Y / n; S.o.cz = Z / n;
        S.o.rmax = R;
        S.o.floor2 = ens_r2_floor(Gm);
        S.xmax_bits = 0;
    }
    __syncthreads();
    float xm = 0.f;
    for (int i = t; i < n; i += T) {  // the thread's own rows, as it wrote them
        const double4 p = pos[i];
        xm = fmaxf(xm, fmaxf(fabsf((float)(p.x - S.o.cx)), fmaxf(fabsf((float)(p.y - S.o.cy)), fabsf((float)(p.z - S.o.cz)))));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) xm = fmaxf(xm, __shfl_xor_sync(0xffffffffu, xm, o));
    if (lane == 0) atomicMax(&S.xmax_bits, __float_as_int(xm));
    __syncthreads();
    if (t == 0) {
        // Bound on the FP32 error of a staged separation: each staged coordinate is within
        // 2^-24 |X| of its FP64 value, so a separation is off by at most sqrt(3) 2^-23 xmax
        // (plus its own relative rounding, covered by the factor on the reach); 2^-21 xmax
        // keeps a factor 2 of room.  Every pair the FP64 overlap test would merge is flagged.
        S.o.slack = __int_as_float(S.xmax_bits) * 0x1p-21f;
        *out = S.o;
    }
    __syncthreads();
}

// Stages a system: FP32 relative positions and G m (padded to an even count, far and massless).
__device__ __forceinline__ void ens_stage(int n, double G, const EnsInfo &f, const double4 *pos, float *sx, float *sy,
                                          float *sz, float *sm) {
    for (int i = threadIdx.x; i < ((n + 1) & ~1); i += blockDim.x) {
        if (i < n) {
            const double4 p = pos[i];
            sx[i] = (float)(p.x - f.cx); sy[i] = (float)(p.y - f.cy); sz[i] = (float)(p.z - f.cz);
            sm[i] = (float)(G * p.w);
        } else {
            sx[i] = 1e30f; sy[i] = 1e30f; sz[i] = 1e30f; sm[i] = 0.f;
        }
    }
}

// The opening half kick and drift (with pre) and the frame of every system.
__global__ void ens_begin_kernel(EnsArgs a) {
    __shared__ EnsBeginSmem S;
    const int s = a.order[blockIdx.x];
    const int64_t b0 = a.off[s];
    ens_begin(a.cnt[s], a.G, a.h, a.pre, a.pos + b0, a.vel + b0, a.acc + b0, a.rad + b0, a.info + s, S);
}

// One launch = the force and closing half kick of one KDK step (or the initial force alone) for every
// system, its merges and, with pre, the next step's opening half kick and drift.  IB bodies per thread
// (1, 2 or 4; each staged j pair feeds IB bodies, dividing the shared-memory reads per interaction by IB).
template <int IB>
__global__ void __launch_bounds__(IB == 1 ? 512 : 256) ensemble_step_kernel(EnsArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float *sx = reinterpret_cast<float *>(smem_raw);
    float *sy = sx + a.stride;
    float *sz = sy + a.stride;
    float *sm = sz + a.stride;
    __shared__ int sh[8], last_s;
    __shared__ EnsCand cand;
    __shared__ EnsBeginSmem S;
    const int t = threadIdx.x, T = blockDim.x;
    const double h2 = 0.5 * a.h;
    const int2 item = a.items[blockIdx.x];
    const int s = item.x;
    const int64_t b0 = a.off[s];
    double4 *pos = a.pos + b0, *vel = a.vel + b0, *acc = a.acc + b0;
    double *rad = a.rad + b0;
    int n = a.cnt[s];
    // the rows of [row0, row1): each of the first sw threads takes t, t + sw, ...: threads hold IB valid
    // rows except in the last warp, and whole warps past sw sit out
    auto rows = [&](int row0, int row1, const EnsInfo &f, bool kick, EnsCand *list) {
        const int sw = ens_row_threads(row1 - row0, IB);
        if (t < sw)
            ens_force_rows<IB>(row0 + t, sw, row1, (n + 1) & ~1, sx, sy, sz, sm, pos, vel, acc, rad, f.rmax, f.slack, kick,
                               h2, f.floor2, list);
    };
    if (item.y < n) {
        const EnsInfo f = a.info[s];
        ens_stage(n, a.G, f, pos, sx, sy, sz, sm);
        __syncthreads();
        rows(item.y, min(item.y + a.chunk, n), f, a.kick != 0, a.merge ? a.cand + s : nullptr);
    }
    // The last chunk of the system to get here finishes the step: everything the others wrote is visible
    // to it (their fence and count, its count and fence).
    __threadfence();
    __syncthreads();
    if (t == 0) {
        const int chunks = (int)((a.off[s + 1] - b0 + a.chunk - 1) / a.chunk);
        last_s = atomicAdd(&a.arrived[s], 1) == chunks - 1;
    }
    __syncthreads();
    if (!last_s) return;
    __threadfence();
    if (t == 0) a.arrived[s] = 0;
    const int listed = a.merge ? __ldcg(&a.cand[s].n) : 0;
    if (listed) {
        for (int k = t; k < min(listed, kEnsCand); k += T) cand.row[k] = __ldcg(&a.cand[s].row[k]);
        if (t == 0) cand.n = listed;
        __syncthreads();
        if (t == 0) a.cand[s].n = 0;
        const int left = listed <= kEnsCand
                             ? ens_merge_scan_cand(n, pos, vel, acc, rad, a.rest + b0, a.ids + b0, cand, sh)
                             : ens_merge_scan(n, 0, false, pos, vel, acc, rad, a.rest + b0, a.ids + b0, sh);
        if (left != n) {
            if (t == 0) {
                a.cnt[s] = left;
                atomicAdd(a.merged, (unsigned)(n - left));
            }
            n = left;
            // the force at the merged state, so the next step's first half kick uses a(x) of the bodies
            // that remain
            ens_begin(n, a.G, a.h, 0, pos, vel, acc, rad, a.info + s, S);
            ens_stage(n, a.G, S.o, pos, sx, sy, sz, sm);
            __syncthreads();
            for (int base = 0; base < n; base += IB * T) rows(base, min(base + IB * T, n), S.o, false, nullptr);
            __threadfence_block();
            __syncthreads();
        }
    }
    if (a.pre) ens_begin(n, a.G, a.h, 1, pos, vel, acc, rad, a.info + s, S);
}

// Host layout (x3 | v3 | a3 | m | r | rest, nb bodies) to the device arrays and back.
__global__ void ens_pack_kernel(const int64_t *off, int64_t nb, const double *io, int has_v, int has_r, int has_rest,
                                double4 *pos, double4 *vel, double4 *acc, double *rad, double *rest, int32_t *ids) {
    const double *x3 = io, *v3 = io + 3 * nb, *m = io + 9 * nb, *r = io + 10 * nb, *e = io + 11 * nb;
    const int64_t b = off[blockIdx.x];
    for (int64_t i = b + threadIdx.x; i < off[blockIdx.x + 1]; i += blockDim.x) {
        pos[i] = make_double4(x3[3 * i], x3[3 * i + 1], x3[3 * i + 2], m[i]);
        vel[i] = has_v ? make_double4(v3[3 * i], v3[3 * i + 1], v3[3 * i + 2], 0.0) : make_double4(0, 0, 0, 0);
        acc[i] = make_double4(0, 0, 0, 0);
        rad[i] = has_r ? r[i] : 0.0;
        rest[i] = has_rest ? e[i] : 1.0;
        ids[i] = (int32_t)(i - b);
    }
}

__global__ void ens_unpack_kernel(int64_t nb, const double4 *pos, const double4 *vel, const double4 *acc, const double *rad,
                                  const double *rest, double *io) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nb) return;
    double *x3 = io, *v3 = io + 3 * nb, *a3 = io + 6 * nb;
    const double4 p = pos[i], v = vel[i], a = acc[i];
    x3[3 * i] = p.x; x3[3 * i + 1] = p.y; x3[3 * i + 2] = p.z;
    v3[3 * i] = v.x; v3[3 * i + 1] = v.y; v3[3 * i + 2] = v.z;
    a3[3 * i] = a.x; a3[3 * i + 1] = a.y; a3[3 * i + 2] = a.z;
    io[9 * nb + i] = p.w;
    io[10 * nb + i] = rad[i];
    io[11 * nb + i] = rest[i];
}

// The kernel for ib bodies per thread (1, 2 or 4).
template <typename F>
void with_ens_kernel(int ib, F &&f) {
    if (ib == 4) f(ensemble_step_kernel<4>);
    else if (ib == 2) f(ensemble_step_kernel<2>);
    else f(ensemble_step_kernel<1>);
}

int ens_smem_bytes(int max_n) { return 4 * ens_stride(max_n) * (int)sizeof(float); }

}  // namespace gtd

using namespace gtd;

static HostSpans ens_spans(const gtd_ensemble *e, const double *m, const double *r, const double *rest, const double *x3,
                           const double *v3, const double *a3) {
    HostSpans o;
    const int64_t nb = e->n_bodies;
    auto add = [&](const double *host, int64_t at, int64_t words) {
        if (host) o.add(host, e->io + at * nb, sizeof(double) * (size_t)(words * nb));
    };
    add(x3, 0, 3);
    add(v3, 3, 3);
    add(a3, 6, 3);
    add(m, 9, 1);
    add(r, 10, 1);
    add(rest, 11, 1);
    return o;
}

static void ens_release_graph(gtd_ensemble *e);

static void ens_release(gtd_ensemble *e) {
    ens_release_graph(e);
    cudaFree(e->items); cudaFree(e->cand); cudaFree(e->info); cudaFree(e->arrived);
    e->items = nullptr; e->cand = nullptr; e->info = nullptr; e->arrived = nullptr;
    e->items_for = 0;
    cudaFree(e->io);
    e->io = nullptr;
    cudaFree(e->off); cudaFree(e->cnt); cudaFree(e->order); cudaFree(e->pos); cudaFree(e->vel); cudaFree(e->acc);
    cudaFree(e->rad); cudaFree(e->rest); cudaFree(e->ids); cudaFree(e->merged);
    e->off = nullptr; e->cnt = nullptr; e->order = nullptr; e->pos = e->vel = e->acc = nullptr;
    e->rad = e->rest = nullptr; e->ids = nullptr; e->merged = nullptr;
}

static EnsArgs ens_args(const gtd_ensemble *e, int kick, int pre) {
    return EnsArgs{e->off, e->cnt, e->order, e->items, e->pos, e->vel, e->acc, e->rad, e->rest, e->ids, e->cand, e->info,
                   e->arrived, e->G, e->dt, kick, pre, e->merge, e->threads * e->ib, ens_stride(e->max_n), e->merged};
}

static void ens_release_graph(gtd_ensemble *e) {
    if (e->graph) cudaGraphExecDestroy(e->graph);
    e->graph = nullptr;
}

// CTA size and bodies per thread for an ensemble nobody configured.  128 threads: the smallest items,
// for balance and latency, unless systems are so large that staging them for 128 or 256 rows shows.  Two
// bodies per thread (fewer shared-memory reads) once that still leaves two rounds of CTAs, 4 per SM.
// Steps in us on B200, 128 x 1 / 128 x 2 / 256 x 1: 4096 systems of up to 2048 bodies 3012 / 2763 / 3106,
// 512 of them 395 / 376 / 402, 128 of them 125 / 140 / 127, 512 of up to 256 19 / 22 / 22, 8 of up to 8192
// 446 / 395 / 350.
static void ens_default(gtd_ensemble *e) {
    e->threads = e->max_n > 4096 ? 256 : 128;
    int64_t items = 0;
    for (int64_t s = 0; s < e->n_sys; ++s) {
        const int64_t n = e->off_h[(size_t)s + 1] - e->off_h[(size_t)s];
        items += (n + 2 * e->threads - 1) / (2 * e->threads);
    }
    e->ib = items >= 8 * 148 ? 2 : 1;
}

// The items for the present CTA size and bodies per thread.
static int ens_prepare(gtd_ensemble *e) {
    const int key = e->threads * 4 + e->ib;
    if (e->items_for == key) return GTD_OK;
    ens_release_graph(e);
    const int chunk = e->threads * e->ib;
    std::vector<int2> items;
    for (int32_t s : e->order_h)
        for (int64_t r = 0; r < e->off_h[(size_t)s + 1] - e->off_h[(size_t)s]; r += chunk)
            items.push_back(make_int2(s, (int)r));
    GTD_CUDA(cudaStreamSynchronize(e->stream));  // no launch reads the old items any more
    cudaFree(e->items);
    e->items = nullptr;
    e->items_for = 0;
    GTD_CUDA(cudaMalloc(&e->items, sizeof(int2) * std::max<size_t>(items.size(), 1)));
    GTD_CUDA(cudaMemcpyAsync(e->items, items.data(), sizeof(int2) * items.size(), cudaMemcpyHostToDevice, e->stream));
    GTD_CUDA(cudaStreamSynchronize(e->stream));
    e->n_items = (int64_t)items.size();
    e->items_for = key;
    return GTD_OK;
}

static int ens_open(gtd_ensemble *e, int pre) {
    ens_begin_kernel<<<(unsigned)e->n_sys, 256, 0, e->stream>>>(ens_args(e, 0, pre));
    GTD_CHECK_LAUNCH();
    return GTD_OK;
}

static int ens_launch(gtd_ensemble *e, int kick, int pre) {
    if (e->n_items > 0) {
        const EnsArgs a = ens_args(e, kick, pre);
        with_ens_kernel(e->ib, [&](auto k) {
            k<<<(unsigned)e->n_items, e->threads, ens_smem_bytes(e->max_n), e->stream>>>(a);
        });
        GTD_CHECK_LAUNCH();
    }
    e->launches += 1;
    return GTD_OK;
}

// Captures `steps` KDK steps, each opening the next, into a CUDA graph.
static int ens_build_graph(gtd_ensemble *e, int steps) {
    ens_release_graph(e);
    cudaGraph_t g;
    GTD_CUDA(cudaStreamBeginCapture(e->stream, cudaStreamCaptureModeThreadLocal));
    int rc = GTD_OK;
    const uint64_t before = e->launches;
    for (int k = 0; k < steps && !rc; ++k) rc = ens_launch(e, 1, 1);
    cudaError_t ce = cudaStreamEndCapture(e->stream, &g);
    e->launches = before;  // captured, not launched
    if (rc) return rc;
    if (ce != cudaSuccess) return cuda_fail(ce, "cudaStreamEndCapture", __FILE__, __LINE__);
    ce = cudaGraphInstantiate(&e->graph, g, 0);
    cudaGraphDestroy(g);
    if (ce != cudaSuccess) return cuda_fail(ce, "cudaGraphInstantiate", __FILE__, __LINE__);
    e->graph_steps = steps;
    e->graph_threads = e->threads * 4 + e->ib;
    return GTD_OK;
}

static int ens_steps(gtd_ensemble *e, uint64_t steps) {
    int rc = ens_prepare(e);
    if (rc) return rc;
    if (!e->begun) {
        rc = ens_open(e, 0);
        if (!rc) rc = ens_launch(e, 0, 1);  // initial accelerations (and add-time merges)
        if (rc) return rc;
        e->begun = true;
    } else if ((rc = ens_open(e, 1))) {
        return rc;
    }
    const int chunk = 16;
    if (steps > (uint64_t)chunk) {  // the last step does not open another
        if (!e->graph || e->graph_steps != chunk || e->graph_threads != e->threads * 4 + e->ib) {
            rc = ens_build_graph(e, chunk);
            if (rc) return rc;
        }
        while (steps > (uint64_t)chunk) {
            GTD_CUDA(cudaGraphLaunch(e->graph, e->stream));
            e->launches += chunk;
            steps -= chunk;
        }
    }
    for (uint64_t k = 0; k < steps; ++k) {
        rc = ens_launch(e, 1, k + 1 < steps ? 1 : 0);
        if (rc) return rc;
    }
    return GTD_OK;
}

static int ens_upload(gtd_ensemble *e, int64_t n_systems, const int64_t *offsets, const double *m, const double *r,
                      const double *rest, const double *x3, const double *v3);

extern "C" {

int gtd_ensemble_create(gtd_ensemble **out, int device) {
    if (!out) return fail(GTD_ERR_INVALID_ARGUMENT, "out is NULL");
    *out = nullptr;
    int nd = 0;
    if (cudaGetDeviceCount(&nd) != cudaSuccess || nd == 0) {
        cudaGetLastError();
        return fail(GTD_ERR_NO_DEVICE, "no CUDA device available");
    }
    if (device < 0 || device >= nd) return fail(GTD_ERR_INVALID_ARGUMENT, "device %d out of range", device);
    GTD_CUDA(cudaSetDevice(device));
    gtd_ensemble *e = new (std::nothrow) gtd_ensemble();
    if (!e) return fail(GTD_ERR_OUT_OF_MEMORY, "host allocation failed");
    e->device = device;
    GTD_CUDA(cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking));
    GTD_CUDA(cudaEventCreate(&e->ev0));
    GTD_CUDA(cudaEventCreate(&e->ev1));
    for (int ib : {1, 2, 4}) {
        cudaError_t c = cudaSuccess;
        with_ens_kernel(ib, [&](auto k) {
            c = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, ens_smem_bytes(kEnsMaxN));
        });
        GTD_CUDA(c);
    }
    *out = e;
    return GTD_OK;
}

int gtd_ensemble_destroy(gtd_ensemble *e) {
    if (!e) return GTD_OK;
    cudaSetDevice(e->device);
    cudaStreamSynchronize(e->stream);
    ens_release(e);
    release_host_ring(e->host_ring);
    cudaEventDestroy(e->ev0);
    cudaEventDestroy(e->ev1);
    cudaStreamDestroy(e->stream);
    delete e;
    return GTD_OK;
}

int gtd_ensemble_set_params(gtd_ensemble *e, double G, double dt, int merge) {
    if (!e) return fail(GTD_ERR_INVALID_ARGUMENT, "ensemble is NULL");
    if (!(dt > 0)) return fail(GTD_ERR_INVALID_ARGUMENT, "Time-step cannot be zero or negative.");
    e->G = G;
    e->dt = dt;
    e->merge = merge ? 1 : 0;
    ens_release_graph(e);
    return GTD_OK;
}

int gtd_ensemble_upload(gtd_ensemble *e, int64_t n_systems, const int64_t *offsets, const double *m,
                        const double *r, const double *rest, const double *x3, const double *v3) {
    if (!e) return fail(GTD_ERR_INVALID_ARGUMENT, "ensemble is NULL");
    if (n_systems < 0 || (n_systems > 0 && (!offsets || !m || !x3)))
        return fail(GTD_ERR_INVALID_ARGUMENT, "bad ensemble description");
    cudaSetDevice(e->device);
    ens_release(e);
    int rc;
    try {
        rc = ens_upload(e, n_systems, offsets, m, r, rest, x3, v3);
    } catch (const std::bad_alloc &) {
        rc = fail(GTD_ERR_OUT_OF_MEMORY, "host allocation failed");
    }
    if (rc) {  // what was there is gone: no systems
        cudaStreamSynchronize(e->stream);
        ens_release(e);
        e->n_sys = e->n_bodies = 0;
    }
    return rc;
}

int gtd_ensemble_evolve(gtd_ensemble *e, uint64_t steps, int64_t *elapsed_ns) {
    if (!e) return fail(GTD_ERR_INVALID_ARGUMENT, "ensemble is NULL");
    if (elapsed_ns) *elapsed_ns = 0;
    if (e->n_sys == 0 || steps == 0) return GTD_OK;
    cudaSetDevice(e->device);
    GTD_CUDA(cudaEventRecord(e->ev0, e->stream));
    int rc = ens_steps(e, steps);
    if (rc) return rc;
    GTD_CUDA(cudaEventRecord(e->ev1, e->stream));
    GTD_CUDA(cudaEventSynchronize(e->ev1));
    float ms = 0.f;
    GTD_CUDA(cudaEventElapsedTime(&ms, e->ev0, e->ev1));
    if (elapsed_ns) *elapsed_ns = (int64_t)((double)ms * 1e6);
    return GTD_OK;
}

int gtd_ensemble_counts(gtd_ensemble *e, int64_t *counts, uint64_t *merges, uint64_t *launches) {
    if (!e) return fail(GTD_ERR_INVALID_ARGUMENT, "ensemble is NULL");
    cudaSetDevice(e->device);
    GTD_CUDA(cudaStreamSynchronize(e->stream));
    if (counts && e->n_sys) {
        std::vector<int32_t> c((size_t)e->n_sys);
        GTD_CUDA(cudaMemcpy(c.data(), e->cnt, sizeof(int32_t) * c.size(), cudaMemcpyDeviceToHost));
        for (int64_t s = 0; s < e->n_sys; ++s) counts[s] = c[(size_t)s];
    }
    if (merges) {
        unsigned w = 0;
        if (e->merged) GTD_CUDA(cudaMemcpy(&w, e->merged, sizeof w, cudaMemcpyDeviceToHost));
        *merges = w;
    }
    if (launches) *launches = e->launches;
    return GTD_OK;
}

int gtd_ensemble_download(gtd_ensemble *e, double *m, double *r, double *rest, double *x3, double *v3,
                          double *a3) {
    if (!e) return fail(GTD_ERR_INVALID_ARGUMENT, "ensemble is NULL");
    cudaSetDevice(e->device);
    GTD_CUDA(cudaStreamSynchronize(e->stream));
    const int64_t nb = e->n_bodies;
    if (!nb) return GTD_OK;
    ens_unpack_kernel<<<(unsigned)((nb + 255) / 256), 256, 0, e->stream>>>(nb, e->pos, e->vel, e->acc, e->rad, e->rest,
                                                                          e->io);
    GTD_CHECK_LAUNCH();
    return copy_to_host(e->host_ring, e->device, e->stream, ens_spans(e, m, r, rest, x3, v3, a3));
}

int gtd_ensemble_set_threads(gtd_ensemble *e, int threads) {
    if (!e) return fail(GTD_ERR_INVALID_ARGUMENT, "ensemble is NULL");
    if (threads != 64 && threads != 128 && threads != 256 && threads != 512)
        return fail(GTD_ERR_INVALID_ARGUMENT, "threads must be 64, 128, 256 or 512");
    if (!e->configured || (e->ib > 1 && threads > 256)) e->ib = 1;
    e->threads = threads;
    e->configured = true;
    return GTD_OK;
}

int gtd_ensemble_set_bodies_per_thread(gtd_ensemble *e, int bodies) {
    if (!e) return fail(GTD_ERR_INVALID_ARGUMENT, "ensemble is NULL");
    if (bodies != 1 && bodies != 2 && bodies != 4)
        return fail(GTD_ERR_INVALID_ARGUMENT, "bodies per thread must be 1, 2 or 4");
    if (bodies > 1 && e->threads > 256)
        return fail(GTD_ERR_INVALID_ARGUMENT, "%d bodies per thread need a CTA of at most 256 threads", bodies);
    if (!e->configured) e->threads = 256;
    e->ib = bodies;
    e->configured = true;
    return GTD_OK;
}

int gtd_ensemble_config(const gtd_ensemble *e, int *threads, int *bodies_per_thread) {
    if (!e) return fail(GTD_ERR_INVALID_ARGUMENT, "ensemble is NULL");
    if (threads) *threads = e->threads;
    if (bodies_per_thread) *bodies_per_thread = e->ib;
    return GTD_OK;
}

// Times a few steps for each CTA size and bodies-per-thread choice on a copy of the current state
// (restored afterwards) and keeps the fastest: the project's tile autotuner for the ensemble.
int gtd_ensemble_autotune(gtd_ensemble *e, int *best_threads, double *best_ms) {
    if (!e) return fail(GTD_ERR_INVALID_ARGUMENT, "ensemble is NULL");
    if (e->n_sys == 0) return fail(GTD_ERR_INVALID_ARGUMENT, "autotune needs systems");
    cudaSetDevice(e->device);
    const int64_t nb = e->n_bodies;
    const size_t b4 = sizeof(double4) * (size_t)nb;
    // copies of the state, freed on every return path
    struct Saved {
        double4 *sp = nullptr, *sv = nullptr, *sa = nullptr;
        double *sr = nullptr, *se = nullptr;
        int32_t *si = nullptr, *sc = nullptr;
        ~Saved() {
            cudaFree(sp); cudaFree(sv); cudaFree(sa); cudaFree(sr); cudaFree(se); cudaFree(si); cudaFree(sc);
        }
    } S;
    GTD_CUDA(cudaMalloc(&S.sp, b4)); GTD_CUDA(cudaMalloc(&S.sv, b4)); GTD_CUDA(cudaMalloc(&S.sa, b4));
    GTD_CUDA(cudaMalloc(&S.sr, 8 * (size_t)nb)); GTD_CUDA(cudaMalloc(&S.se, 8 * (size_t)nb));
    GTD_CUDA(cudaMalloc(&S.si, 4 * (size_t)nb)); GTD_CUDA(cudaMalloc(&S.sc, 4 * (size_t)e->n_sys));
    double4 *sp = S.sp, *sv = S.sv, *sa = S.sa;
    double *sr = S.sr, *se = S.se;
    int32_t *si = S.si, *sc = S.sc;
    auto save = [&](bool back) -> int {
        auto cp = [&](void *dst, void *src, size_t bytes) { return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, e->stream); };
        cudaError_t c = cudaSuccess;
        if (!back) {
            c = cp(sp, e->pos, b4); if (!c) c = cp(sv, e->vel, b4); if (!c) c = cp(sa, e->acc, b4);
            if (!c) c = cp(sr, e->rad, 8 * nb); if (!c) c = cp(se, e->rest, 8 * nb); if (!c) c = cp(si, e->ids, 4 * nb);
            if (!c) c = cp(sc, e->cnt, 4 * e->n_sys);
        } else {
            c = cp(e->pos, sp, b4); if (!c) c = cp(e->vel, sv, b4); if (!c) c = cp(e->acc, sa, b4);
            if (!c) c = cp(e->rad, sr, 8 * nb); if (!c) c = cp(e->rest, se, 8 * nb); if (!c) c = cp(e->ids, si, 4 * nb);
            if (!c) c = cp(e->cnt, sc, 4 * e->n_sys);
        }
        return c == cudaSuccess ? GTD_OK : cuda_fail(c, "autotune state copy", __FILE__, __LINE__);
    };
    int rc = save(false);
    const bool was_begun = e->begun;
    const int orig_threads = e->threads, orig_ib = e->ib;
    const int cands[][2] = {{128, 1}, {256, 1}, {512, 1}, {128, 2}, {256, 2}, {128, 4}, {256, 4}};
    constexpr int kCands = sizeof(cands) / sizeof(cands[0]);
    // Each timing runs kTuneSteps consecutive steps from the saved state, so a candidate is judged on
    // steady stepping rather than on one launch.  The candidates take turns (round robin) so that a
    // clock still ramping up after the upload favours none of them; the first round only warms up.
    constexpr int kTuneSteps = 4, kRounds = 3;
    double per[kCands];
    for (int k = 0; k < kCands; ++k) per[k] = 1e300;
    for (int round = 0; round < kRounds && !rc; ++round) {
        for (int k = 0; k < kCands && !rc; ++k) {
            e->threads = cands[k][0];
            e->ib = cands[k][1];
            if ((rc = ens_prepare(e))) break;
            if ((rc = cudaEventRecord(e->ev0, e->stream) ? GTD_ERR_CUDA : GTD_OK)) break;
            rc = ens_open(e, 1);
            for (int q = 0; q < kTuneSteps && !rc; ++q) rc = ens_launch(e, 1, q + 1 < kTuneSteps ? 1 : 0);
            if (rc) break;
            cudaEventRecord(e->ev1, e->stream);
            cudaEventSynchronize(e->ev1);
            float ms = 0.f;
            cudaEventElapsedTime(&ms, e->ev0, e->ev1);
            if (round > 0) per[k] = std::min(per[k], (double)ms / kTuneSteps);
            rc = save(true);
        }
    }
    if (rc) {  // a failed copy or launch: leave the configuration as it was
        e->threads = orig_threads;
        e->ib = orig_ib;
        e->begun = was_begun;
        cudaStreamSynchronize(e->stream);
        return rc;
    }
    int best = orig_threads, best_ib = orig_ib;  // kept if no timing completed
    double bestv = 1e300;
    for (int k = 0; k < kCands; ++k)
        if (per[k] < bestv) {
            bestv = per[k];
            best = cands[k][0];
            best_ib = cands[k][1];
        }
    e->threads = best;
    e->ib = best_ib;
    e->configured = true;
    e->begun = was_begun;
    GTD_CUDA(cudaStreamSynchronize(e->stream));
    GTD_CUDA(cudaMemset(e->merged, 0, sizeof(unsigned)));
    if (best_threads) *best_threads = best;
    if (best_ms) *best_ms = bestv;
    return GTD_OK;
}

}  // extern "C"

// The systems of an empty handle; after an error some of its buffers may be there.
static int ens_upload(gtd_ensemble *e, int64_t n_systems, const int64_t *offsets, const double *m, const double *r,
                      const double *rest, const double *x3, const double *v3) {
    e->n_sys = n_systems;
    const int64_t none = 0;
    if (!n_systems) offsets = &none;
    e->off_h.assign(offsets, offsets + n_systems + 1);
    const int64_t nb = offsets[n_systems];
    e->n_bodies = nb;
    e->max_n = 0;
    std::vector<int32_t> cnt((size_t)n_systems);
    std::vector<int32_t> &order = e->order_h;
    order.assign((size_t)n_systems, 0);
    for (int64_t s = 0; s < n_systems; ++s) {
        const int64_t k = offsets[s + 1] - offsets[s];
        if (k < 0 || offsets[s] < 0) return fail(GTD_ERR_INVALID_ARGUMENT, "offsets must be non-decreasing from 0");
        if (k > kEnsMaxN) return fail(GTD_ERR_CAPACITY, "system %lld has %lld bodies; the ensemble kernel holds %d",
                                      (long long)s, (long long)k, kEnsMaxN);
        cnt[(size_t)s] = (int32_t)k;
        e->max_n = std::max(e->max_n, (int)k);
    }
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int32_t a, int32_t b) { return cnt[a] > cnt[b]; });
    const int64_t first = offsets[0];  // rows before it belong to no system and read as zero
    for (int64_t i = first; i < nb; ++i)
        if (m[i] < 0) return fail(GTD_ERR_INVALID_ARGUMENT, "negative mass at body %lld", (long long)i);
    const size_t b4 = sizeof(double4) * (size_t)std::max<int64_t>(nb, 1);
    GTD_CUDA(cudaMalloc(&e->off, sizeof(int64_t) * (size_t)(n_systems + 1)));
    GTD_CUDA(cudaMalloc(&e->cnt, sizeof(int32_t) * (size_t)std::max<int64_t>(n_systems, 1)));
    GTD_CUDA(cudaMalloc(&e->order, sizeof(int32_t) * (size_t)std::max<int64_t>(n_systems, 1)));
    GTD_CUDA(cudaMalloc(&e->pos, b4));
    GTD_CUDA(cudaMalloc(&e->vel, b4));
    GTD_CUDA(cudaMalloc(&e->acc, b4));
    GTD_CUDA(cudaMalloc(&e->rad, sizeof(double) * (size_t)std::max<int64_t>(nb, 1)));
    GTD_CUDA(cudaMalloc(&e->rest, sizeof(double) * (size_t)std::max<int64_t>(nb, 1)));
    GTD_CUDA(cudaMalloc(&e->ids, sizeof(int32_t) * (size_t)std::max<int64_t>(nb, 1)));
    GTD_CUDA(cudaMalloc(&e->merged, sizeof(unsigned)));
    const size_t ns = (size_t)std::max<int64_t>(n_systems, 1);
    GTD_CUDA(cudaMalloc(&e->cand, sizeof(EnsCand) * ns));
    GTD_CUDA(cudaMalloc(&e->info, sizeof(EnsInfo) * ns));
    GTD_CUDA(cudaMalloc(&e->arrived, sizeof(int) * ns));
    cudaStream_t st = e->stream;
    GTD_CUDA(cudaMemsetAsync(e->cand, 0, sizeof(EnsCand) * ns, st));
    GTD_CUDA(cudaMemsetAsync(e->arrived, 0, sizeof(int) * ns, st));
    GTD_CUDA(cudaMemcpyAsync(e->off, offsets, sizeof(int64_t) * (size_t)(n_systems + 1), cudaMemcpyHostToDevice, st));
    if (n_systems) {
        GTD_CUDA(cudaMemcpyAsync(e->cnt, cnt.data(), sizeof(int32_t) * cnt.size(), cudaMemcpyHostToDevice, st));
        GTD_CUDA(cudaMemcpyAsync(e->order, order.data(), sizeof(int32_t) * order.size(), cudaMemcpyHostToDevice, st));
    }
    if (nb) {
        GTD_CUDA(cudaMalloc(&e->io, 12 * sizeof(double) * (size_t)nb));
        int rc = copy_to_device(e->host_ring, e->device, e->stream, ens_spans(e, m, r, rest, x3, v3, nullptr));
        if (rc) return rc;
        ens_pack_kernel<<<(unsigned)n_systems, 256, 0, e->stream>>>(e->off, nb, e->io, v3 != nullptr, r != nullptr,
                                                                    rest != nullptr, e->pos, e->vel, e->acc, e->rad,
                                                                    e->rest, e->ids);
        GTD_CHECK_LAUNCH();
        if (first > 0) {
            GTD_CUDA(cudaMemsetAsync(e->pos, 0, sizeof(double4) * (size_t)first, st));
            GTD_CUDA(cudaMemsetAsync(e->vel, 0, sizeof(double4) * (size_t)first, st));
            GTD_CUDA(cudaMemsetAsync(e->acc, 0, sizeof(double4) * (size_t)first, st));
            GTD_CUDA(cudaMemsetAsync(e->rad, 0, sizeof(double) * (size_t)first, st));
            GTD_CUDA(cudaMemsetAsync(e->rest, 0, sizeof(double) * (size_t)first, st));
        }
    }
    GTD_CUDA(cudaMemsetAsync(e->merged, 0, sizeof(unsigned), st));
    GTD_CUDA(cudaStreamSynchronize(st));
    e->begun = false;
    if (!e->configured) ens_default(e);
    return GTD_OK;
}

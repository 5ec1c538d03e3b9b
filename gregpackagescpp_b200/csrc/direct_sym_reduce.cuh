// The partial sums of the unordered-pair kernels: where a batch's slots lie, and the kernel body that
// adds a body's row and column slots.
#pragma once

#include "direct_mixed.cuh"
#include "direct_sym_geom.cuh"

namespace gtd {

// term(0) + .. + term(N - 1), added as a balanced tree (short dependent chains, fixed order).
template <int N, typename F>
__device__ __forceinline__ double sym_tree(F &&term) {
    double v[N];
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = term(k);
#pragma unroll
    for (int h = N / 2; h > 0; h >>= 1)
#pragma unroll
        for (int k = 0; k < h; ++k) v[k] += v[k + h];
    return v[0];
}

// A batch's slots of D words per body.
struct SymSlots {
    SymGeom g;
    const double *rowpart, *colpart;
    int64_t unit0, col0;  // first unit and first column slot of the batch
    int64_t Pa, Pb;       // super-groups of the batch
    const double *base;   // sums of the earlier batches (D arrays of n), or NULL
};

// Buffer: a queue counter per batch | the running sum (where there are several batches) | slots.
struct SymLayout {
    int64_t batches = 0;
    size_t base = 0, slots = 0, bytes = 0;
};

inline SymLayout sym_layout(const SymGeom &g, size_t slot_bytes, int D) {
    SymLayout o;
    size_t most = 0;
    for (int64_t P = 0; P < g.Gs;) {
        const int64_t e = sym_batch_end(g, P, slot_bytes, D);
        most = std::max(most, sym_slot_bytes(g, P, e, D));
        ++o.batches;
        P = e;
    }
    o.base = ((size_t)o.batches * sizeof(unsigned) + 255) / 256 * 256;
    o.slots = o.base + (o.batches > 1 ? ((size_t)D * g.n * sizeof(double) + 255) / 256 * 256 : 0);
    o.bytes = o.slots + most;
    return o;
}

inline SymSlots sym_slots(const SymGeom &g, const SymLayout &lay, const char *mem, int64_t Pa, int64_t Pb, int D) {
    SymSlots r{};
    r.g = g;
    r.unit0 = sym_tri(g, Pa) * sym_block_units(g);
    r.col0 = sym_col_off(g, Pa * g.L * g.s);
    r.rowpart = reinterpret_cast<const double *>(mem + lay.slots);
    r.colpart = r.rowpart + (size_t)((sym_tri(g, Pb) - sym_tri(g, Pa)) * sym_block_units(g)) * D * g.B;
    r.Pa = Pa;
    r.Pb = Pb;
    r.base = Pa > 0 ? reinterpret_cast<const double *>(mem + lay.base) : nullptr;
    return r;
}

// 32 bodies per CTA; warp w takes every kRedWarps-th slot of each body (consecutive bodies read
// consecutive words), compensated; the warps' sums are added in warp order and handed to
// finish(i, sums).  With a thread per body the reads of a small system would queue up behind one
// another (65 us at N = 16384 with four words, against 9).
constexpr int kRedWarps = 8;

template <int D, typename F>
__device__ __forceinline__ void sym_reduce(const SymSlots &a, F &&finish) {
    __shared__ double part[kRedWarps][D][32];
    const SymGeom &g = a.g;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t i0 = (int64_t)blockIdx.x * 32, i = i0 + lane;
    // B, TC and W are multiples of 32: the CTA's bodies share a row block, a tile and a group
    const int64_t b = i0 / g.B, R = i0 / g.W, P = R / g.L, tile = i0 / g.TC;
    const int l = (int)(i0 - b * g.B) + lane, cl = (int)(i0 - tile * g.TC) + lane;
    double s[D], k[D];
#pragma unroll
    for (int d = 0; d < D; ++d) s[d] = k[d] = 0.0;
    if (i < g.n) {
        int64_t rows = 0;  // row slots of the body in this batch
        if (P >= a.Pa && P < a.Pb) rows = (g.Gs - P) * g.q;
        const int64_t per = sym_block_units(g);
        const int64_t u0 = sym_tri(g, P) * per + (b - P * g.L * g.s) * g.q - a.unit0;
#pragma unroll 2
        for (int64_t e = warp; e < rows; e += kRedWarps) {
            const int64_t Q = e / g.q, sub = e - Q * g.q;
            const double *slot = a.rowpart + (size_t)(u0 + Q * per + sub) * D * g.B + l;
#pragma unroll
            for (int d = 0; d < D; ++d) kahan_add(s[d], k[d], slot[d * g.B]);
        }
        const int64_t r0 = a.Pa * g.L * g.s, r1 = min(a.Pb * g.L, R) * g.s;
#pragma unroll 4
        for (int64_t r = r0 + warp; r < r1; r += kRedWarps) {
            const int64_t at = sym_col_off(g, r) - a.col0 + tile - (r / g.s + 1) * g.kw;
            const double *slot = a.colpart + (size_t)at * D * g.TC + cl;
#pragma unroll
            for (int d = 0; d < D; ++d) kahan_add(s[d], k[d], slot[d * g.TC]);
        }
    }
#pragma unroll
    for (int d = 0; d < D; ++d) part[warp][d][lane] = s[d] - k[d];
    __syncthreads();
    if (warp != 0 || i >= g.n) return;
    double v[D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
        double sum = 0.0, comp = 0.0;
        if (a.base) sum = a.base[(size_t)d * g.n + i];
#pragma unroll
        for (int w = 0; w < kRedWarps; ++w) kahan_add(sum, comp, part[w][d][lane]);
        v[d] = sum - comp;
    }
    finish(i, v);
}

}  // namespace gtd

// Decomposition of the direct sum that evaluates each unordered pair once (direct_sym.cu): units,
// partial-sum slots and batches as index arithmetic, without a device.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

namespace gtd {

struct SymGeom {
    int64_t n = 0;
    int B = 0, TC = 0, W = 0;  // bodies per row block, per column tile, per group
    int s = 0, kw = 0;         // row blocks and tiles per group
    int L = 1, q = 1;          // groups joined in a unit's columns, or parts a group's columns are cut into
    int64_t nt = 0, G = 0, Gs = 0;  // tiles, groups, joined groups
};
constexpr size_t kSymSlotBytes = (size_t)5 << 28;  // 1.25 GiB
struct SymShape {
    int i, threads, tile, group;
    double unit = 0.1;  // what a unit costs beside its tiles, in tiles of 64 columns
};

// First unit block (P, P): super-groups P, Q of L groups, Q >= P, in row-major order.
__host__ __device__ __forceinline__ int64_t sym_tri(const SymGeom &g, int64_t P) { return P * g.Gs - P * (P - 1) / 2; }

__host__ __device__ __forceinline__ int64_t sym_block_units(const SymGeom &g) { return (int64_t)g.L * g.s * g.q; }

// First column slot of row block r.
__host__ __device__ __forceinline__ int64_t sym_col_off(const SymGeom &g, int64_t r) {
    const int64_t R = r / g.s;
    const int64_t own = g.nt - (R + 1) * g.kw;  // tiles after the group (not used where none are left)
    return g.s * (R * g.nt - g.kw * R * (R + 1) / 2) + (r - R * g.s) * own;
}

struct SymUnit {
    int64_t r, c0, c1;  // row block, first and past-the-last column tile
};

__host__ __device__ __forceinline__ SymUnit sym_unit(const SymGeom &g, int64_t u) {
    const int64_t per = sym_block_units(g);
    const int64_t b = u / per, rem = u - b * per;
    const double q = (double)(2 * g.Gs + 1);
    int64_t P = (int64_t)floor((q - sqrt(q * q - 8.0 * (double)b)) * 0.5);
    P = P < 0 ? 0 : (P > g.Gs - 1 ? g.Gs - 1 : P);
    while (P > 0 && sym_tri(g, P) > b) --P;
    while (P + 1 < g.Gs && sym_tri(g, P + 1) <= b) ++P;
    const int64_t Q = P + (b - sym_tri(g, P));
    const int64_t row = rem / g.q, sub = rem - row * g.q;
    SymUnit o;
    o.r = P * g.L * g.s + row;
    const int64_t width = (int64_t)g.kw * g.L / g.q;
    const int64_t c = Q * g.L * g.kw + sub * width;
    o.c1 = c + width < g.nt ? c + width : g.nt;
    const int64_t own = (o.r / g.s) * g.kw;
    o.c0 = c > own ? c : own;
    return o;
}

// Bytes of the slots of super-groups [Pa, Pb), D words per body.
inline size_t sym_slot_bytes(const SymGeom &g, int64_t Pa, int64_t Pb, int D = 3) {
    const int64_t units = (sym_tri(g, Pb) - sym_tri(g, Pa)) * sym_block_units(g);
    const int64_t cols = sym_col_off(g, std::min(Pb * g.L, g.G - 1) * g.s) - sym_col_off(g, std::min(Pa * g.L, g.G - 1) * g.s);
    return ((size_t)units * g.B + (size_t)cols * g.TC) * D * sizeof(double);
}

// The end of the batch that starts at super-group Pa: as many as fit `bytes` (at least one).
inline int64_t sym_batch_end(const SymGeom &g, int64_t Pa, size_t bytes, int D = 3) {
    int64_t Pb = Pa + 1;
    while (Pb < g.Gs && sym_slot_bytes(g, Pa, Pb + 1, D) <= bytes) ++Pb;
    return Pb;
}

// The decomposition for n bodies on sms SMs that hold per_sm CTAs each.
inline SymGeom sym_geometry(int64_t n, const SymShape &sh, int sms, int per_sm) {
    SymGeom g;
    g.n = n;
    g.B = sh.i * sh.threads;
    g.TC = sh.tile;
    g.W = sh.group;
    g.s = g.W / g.B;
    g.kw = g.W / g.TC;
    g.nt = (n + g.TC - 1) / g.TC;
    g.G = (n + g.W - 1) / g.W;
    const int64_t ctas = (int64_t)sms * per_sm;
    const int64_t blocks = g.G * (g.G + 1) / 2 * g.s;
    // The columns of a unit: where there are few groups each is cut into q parts.  A unit costs its
    // tiles and sh.unit, an SM runs per_sm units side by side (fewer leave
    // its pipe partly idle), and the SM with the most units sets the time.
    double best = 0.0;
    for (int q = 1; g.kw % q == 0; q *= 2) {
        const double each = (double)((blocks * q + sms - 1) / sms);
        const double side = std::min<double>(each, per_sm);
        const double cost = each * ((double)(g.kw / q) * g.TC / 64 + sh.unit) * (side + per_sm) / (2.0 * side);
        if (q == 1 || cost < best) {
            best = cost;
            g.q = q;
        }
    }
    // where there are many, L groups are joined (fewer row slots), keeping some 48 units per CTA and
    // batches that are small against their bound
    g.Gs = g.G;
    while (g.q == 1 && blocks / (2 * g.L) >= 48 * ctas && sym_slot_bytes(g, 0, 1) < kSymSlotBytes / 16) {
        g.L *= 2;
        g.Gs = (g.G + g.L - 1) / g.L;
    }
    return g;
}

}  // namespace gtd

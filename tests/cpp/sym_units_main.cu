// The index arithmetic of the unordered-pair direct sum, checked on the host: every (row block, column
// tile) pair at or after the row block's own group belongs to exactly one unit, every column slot is
// written once and read by exactly the bodies of its tile, and the slots of a batch fit their bytes.
#include <cstdio>
#include <vector>

#include "direct_sym_geom.cuh"

using namespace gtd;

static int check(const SymGeom &g, size_t bytes) {
    const int64_t nb = (g.n + g.B - 1) / g.B, per = sym_block_units(g);
    std::vector<char> cover((size_t)(nb * g.nt), 0);
    for (int64_t Pa = 0; Pa < g.Gs;) {
        const int64_t Pb = sym_batch_end(g, Pa, bytes);
        const int64_t u0 = sym_tri(g, Pa) * per, u1 = sym_tri(g, Pb) * per, col0 = sym_col_off(g, Pa * g.L * g.s);
        const int64_t cols = ((int64_t)(sym_slot_bytes(g, Pa, Pb) / 24) - (u1 - u0) * g.B) / g.TC;
        if (Pb > Pa + 1 && sym_slot_bytes(g, Pa, Pb) > bytes) return 1;
        std::vector<int64_t> wrote((size_t)cols, -1);  // the tile each column slot holds
        for (int64_t u = u0; u < u1; ++u) {
            const SymUnit o = sym_unit(g, u);
            if (o.r < 0) return 2;
            if (o.r * g.B >= g.n) continue;
            for (int64_t t = o.c0; t < o.c1; ++t) {
                if (t < 0 || t >= g.nt || cover[(size_t)(o.r * g.nt + t)]++) return 3;
                const int64_t own_end = (o.r / g.s + 1) * g.kw;
                if (t < own_end) continue;
                const int64_t at = sym_col_off(g, o.r) - col0 + t - own_end;
                if (at < 0 || at >= cols || wrote[(size_t)at] != -1) return 4;
                wrote[(size_t)at] = t;
            }
        }
        std::vector<char> read((size_t)cols, 0);
        for (int64_t t = 0; t < g.nt; ++t) {  // the row and column slots the reduction takes for a tile's bodies
            const int64_t i = t * g.TC, b = i / g.B, R = i / g.W, P = R / g.L;
            if (P >= Pa && P < Pb)
                for (int64_t e = 0; e < (g.Gs - P) * g.q; ++e) {
                    const int64_t u = sym_tri(g, P) * per + (b - P * g.L * g.s) * g.q + (e / g.q) * per + e % g.q;
                    if (u < u0 || u >= u1 || sym_unit(g, u).r != b) return 5;
                }
            for (int64_t r = Pa * g.L * g.s; r < std::min(Pb * g.L, R) * g.s; ++r) {
                const int64_t at = sym_col_off(g, r) - col0 + t - (r / g.s + 1) * g.kw;
                if (at < 0 || at >= cols || wrote[(size_t)at] != t) return 6;
                read[(size_t)at] = 1;
            }
        }
        for (int64_t k = 0; k < cols; ++k)
            if ((wrote[(size_t)k] != -1) != (read[(size_t)k] != 0)) return 7;
        Pa = Pb;
    }
    for (int64_t r = 0; r < nb; ++r)
        for (int64_t t = 0; t < g.nt; ++t)
            if (cover[(size_t)(r * g.nt + t)] != (t >= (r / g.s) * g.kw)) return 8;
    return 0;
}

int main() {
    const SymShape shapes[] = {{4, 128, 64, 512}, {4, 128, 128, 512}, {4, 128, 128, 1024}, {2, 128, 64, 512}};
    int checked = 0;
    for (const SymShape &sh : shapes)
        for (int64_t n : {1, 2, 63, 64, 65, 511, 512, 513, 1024, 1025, 4097, 8191, 12345, 30001})
            for (int sms : {3, 37, 148})
                for (int per_sm : {1, 3})
                    for (size_t bytes : {kSymSlotBytes, (size_t)3 << 20}) {
                        const SymGeom g = sym_geometry(n, sh, sms, per_sm);
                        if (int rc = check(g, bytes)) {
                            std::printf("n=%lld shape %d/%d sms=%d per_sm=%d: %d\n", (long long)n, sh.tile, sh.group, sms,
                                        per_sm, rc);
                            return 1;
                        }
                        ++checked;
                    }
    std::printf("ok %d\n", checked);
    return 0;
}

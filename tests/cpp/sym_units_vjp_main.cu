// The unordered-pair index arithmetic (sym_units_main.cu) for the shape and the four words per body of the
// adjoint's VJP: the same cover of pairs and slots, and the batches' slots inside their buffer.
#define main sym_units_main
#include "sym_units_main.cu"
#undef main

#include "direct_sym_reduce.cuh"

// Row and column slots of each batch lie in order inside the buffer that sym_layout sizes.
static int layout(const SymGeom &g, size_t bytes, int D) {
    const SymLayout lay = sym_layout(g, bytes, D);
    if (lay.base < (size_t)lay.batches * sizeof(unsigned) || lay.slots < lay.base) return 20;
    if (lay.batches > 1 && lay.slots - lay.base < (size_t)D * g.n * sizeof(double)) return 21;
    const char *mem = reinterpret_cast<const char *>((uintptr_t)1 << 20);
    int64_t batch = 0;
    for (int64_t Pa = 0; Pa < g.Gs; ++batch) {
        const int64_t Pb = sym_batch_end(g, Pa, bytes, D), per = sym_block_units(g);
        const SymSlots s = sym_slots(g, lay, mem, Pa, Pb, D);
        const int64_t units = (sym_tri(g, Pb) - sym_tri(g, Pa)) * per;
        int64_t cols = 0;  // column slots that the batch's units write
        for (int64_t u = s.unit0; u < s.unit0 + units; ++u) {
            const SymUnit o = sym_unit(g, u);
            if (o.r * g.B >= g.n) continue;
            for (int64_t t = std::max(o.c0, (o.r / g.s + 1) * g.kw); t < o.c1; ++t) {
                const int64_t at = sym_col_off(g, o.r) - s.col0 + t - (o.r / g.s + 1) * g.kw;
                if (at < 0) return 22;
                cols = std::max(cols, at + 1);
            }
        }
        const char *row = reinterpret_cast<const char *>(s.rowpart), *col = reinterpret_cast<const char *>(s.colpart);
        if (row != mem + lay.slots || col != row + (size_t)units * D * g.B * sizeof(double)) return 23;
        if ((size_t)(col - mem) + (size_t)cols * D * g.TC * sizeof(double) > lay.bytes) return 24;
        if ((Pa > 0) != (s.base != nullptr)) return 25;
        Pa = Pb;
    }
    return batch == lay.batches ? 0 : 26;
}

int main() {
    const SymShape vjp{2, 128, 64, 256};
    int checked = 0;
    for (int64_t n : {1, 2, 63, 64, 65, 255, 256, 257, 512, 513, 3401, 4097, 8191, 12345, 30001})
        for (int sms : {3, 37, 148})
            for (int per_sm : {1, 3})
                for (size_t bytes : {kSymSlotBytes, (size_t)5 << 20, (size_t)3 << 20}) {
                    const SymGeom g = sym_geometry(n, vjp, sms, per_sm);
                    int rc = check(g, bytes);
                    for (int D = 3; D <= 4 && !rc; ++D) rc = layout(g, bytes, D);
                    if (rc) return std::printf("n=%lld sms=%d per_sm=%d bytes=%zu: %d\n", (long long)n, sms, per_sm, bytes, rc), 1;
                    ++checked;
                }
    std::printf("ok %d\n", checked);
    return 0;
}

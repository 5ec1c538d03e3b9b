// The rows that the threads of the ensemble's force loop read, checked on the host: every read lies in the
// system's staged rows, the rows of a thread that has them are its own, and each row is taken once.
#include <cstdio>
#include <vector>

#include "ensemble_rows.cuh"

using namespace gtd;

int main() {
    int checked = 0;
    for (int n = 1; n <= 600; ++n)
        for (int ib : {1, 2, 4})
            for (int threads : {64, 128, 256, 512}) {
                if (ib > 1 && threads > 256) continue;
                const int chunk = threads * ib;
                std::vector<int> taken((size_t)n, 0);
                for (int row0 = 0; row0 < n; row0 += chunk) {
                    const int row1 = std::min(row0 + chunk, n), sw = ens_row_threads(row1 - row0, ib);
                    if (sw > threads || sw % 32) return std::printf("n=%d ib=%d threads=%d: %d threads\n", n, ib, threads, sw), 1;
                    for (int t = 0; t < sw; ++t)
                        for (int b = 0; b < ib; ++b) {
                            const int r0 = row0 + t, i = r0 + b * sw, at = ens_staged_row(i, r0, row1);
                            if (at < 0 || at >= n || at >= ens_stride(n) || (i < row1 && at != i))
                                return std::printf("n=%d ib=%d threads=%d t=%d b=%d reads row %d\n", n, ib, threads, t, b, at), 1;
                            if (i < row1) ++taken[(size_t)i];
                            ++checked;
                        }
                }
                for (int c : taken)
                    if (c != 1) return std::printf("n=%d ib=%d threads=%d: a row taken %d times\n", n, ib, threads, c), 1;
            }
    std::printf("ok %d\n", checked);
    return 0;
}

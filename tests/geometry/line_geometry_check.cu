// Host check (no GPU) of the line-form stage kernel's shared-memory positions (vlasov_stage_line.cuh), for
// every order, both precisions, every line of every thread (those past the last one too) and every number
// of elements in a tile: a v line's values and its upwind trace lie in the tile buffer, in the line's own
// row, and the trace is the neighbouring element's node or the one kept beside the tile.
#include <cstdio>

#include "vlasov_stage_line.cuh"

static int failures = 0;

static void expect(bool ok, const char *what, int n, int es, int r, int b, int nb) {
    if (ok) return;
    if (failures++ < 20) std::printf("FAIL n=%d element=%dB row=%d b=%d nb=%d: %s\n", n, es, r, b, nb, what);
}

template <int N, typename T>
void check() {
    using G = vl::LineGeom<N, T>;
    const int es = (int)sizeof(T);
    for (int tid = 0; tid < G::THREADS; ++tid)
        for (int s = 0; s < G::L; ++s) {
            // as in the kernel: line l of the thread
            const int l = tid + s * G::THREADS;
            const bool has = l < G::LINES;
            const int r = has ? l % (N * N) : 0, b = has ? l / (N * N) : 1 << 20;
            for (int nb = 1; nb <= G::EPT; ++nb) {
                const int bb = vl::line_elem(b, nb), p = r * G::W + bb * N;
                expect(bb == (b < nb ? b : 0), "element", N, es, r, b, nb);
                expect(p % G::VEC == 0 && p + N <= r * G::W + nb * N && p + N <= G::BUF, "values", N, es, r, b, nb);
                for (int pos = 0; pos < 2; ++pos) {
                    if (vl::line_trace_beside(bb, nb, pos != 0)) continue;   // (r < N N: a row of the halo buffer)
                    const int to = p + (pos ? -1 : N);
                    expect(to >= r * G::W && to < r * G::W + nb * N, "trace in its row", N, es, r, b, nb);
                }
                if (b < nb) {
                    expect(vl::line_trace_beside(bb, nb, true) == (b == 0), "left trace", N, es, r, b, nb);
                    expect(vl::line_trace_beside(bb, nb, false) == (b == nb - 1), "right trace", N, es, r, b, nb);
                }
            }
        }
}

template <typename T>
void all() {
    check<1, T>();
    check<2, T>();
    check<3, T>();
    check<4, T>();
    check<5, T>();
    check<6, T>();
    check<7, T>();
    check<8, T>();
    check<9, T>();
    check<10, T>();
}

int main() {
    all<double>();
    all<float>();
    if (failures) {
        std::printf("%d failures\n", failures);
        return 1;
    }
    std::printf("ALL OK\n");
    return 0;
}

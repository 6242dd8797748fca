// tridiag_lowest (mcpi_b200/csrc/tridiag.cpp) against tridiag_eig on random and
// on graded tridiagonals: the same lowest value, the same vector with its sign;
// and the host memory it holds at most, counted in operator new.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <random>
#include <vector>

#include "../../mcpi_b200/csrc/tridiag.cpp"

static size_t g_held = 0, g_peak = 0;
static size_t g_limit = (size_t)-1;   // operator new throws beyond this

void *operator new(size_t n)
{
    if (n > g_limit - g_held) throw std::bad_alloc();
    size_t *p = static_cast<size_t *>(std::malloc(n + 16));
    if (!p) throw std::bad_alloc();
    *p = n;
    g_held += n;
    if (g_held > g_peak) g_peak = g_held;
    return p + 2;
}
void operator delete(void *p) noexcept
{
    if (!p) return;
    size_t *q = static_cast<size_t *>(p) - 2;
    g_held -= *q;
    std::free(q);
}
void operator delete(void *p, size_t) noexcept { operator delete(p); }

int main()
{
    std::mt19937_64 rng(5);
    std::normal_distribution<double> normal;
    for (int n : {1, 2, 3, 10, 57, 375, 600})
        for (int kind = 0; kind < 3; ++kind) {
            std::vector<double> d(n), e(n > 1 ? n - 1 : 1), z((size_t)n * n), v(n);
            for (int k = 0; k < n; ++k) d[k] = kind == 0 ? normal(rng) : kind == 1 ? 50.0 + 40.0 * std::cos(k) : 1.0;
            for (int k = 0; k + 1 < n; ++k) e[k] = kind == 2 ? 0.5 / (k + 1) : std::fabs(normal(rng)) + 0.1;
            std::vector<double> d1 = d, d2 = d;
            if (mcpi::tridiag_eig(n, d1.data(), e.data(), z.data())) return std::printf("eig n=%d\n", n), 1;
            const size_t before = g_held;
            g_peak = g_held;
            double E = 0.0;
            if (mcpi::tridiag_lowest(n, d2.data(), e.data(), &E, v.data())) return std::printf("lowest n=%d\n", n), 1;
            // held: two factors per rotation (1.0 n^2 rotations of a Lanczos matrix, up to
            // 1.4 n^2 of a random one), one block not yet full, and by sweep and by block
            // what a vector that doubles holds at most (twice over while it grows)
            size_t rot = 0, sweeps = 1;
            const size_t peak = g_peak - before;
            {
                std::vector<double> d3 = d, e3(n, 0.0);
                for (int k = 0; k + 1 < n; ++k) e3[k] = e[k];
                int last = -1;
                mcpi::ql(n, d3.data(), e3.data(), [&](int i, double, double) {
                    ++rot;
                    sweeps += i != last - 1;
                    last = i;
                });
            }
            if (peak > 16 * (rot + 1024) + 3 * (16 * sweeps + 8 * (rot / 1024 + 1)) + 8 * (size_t)n + 256)
                return std::printf("n=%d kind=%d: %zu bytes = %.1f n^2\n", n, kind, peak, (double)peak / n / n), 1;
            if (E != d1[0]) return std::printf("E n=%d kind=%d\n", n, kind), 1;
            // near ties the lowest vector is only as good as the gap
            const double gap = n > 1 ? d1[1] - d1[0] : 1.0, tol = 1e-12 + 1e-13 * std::sqrt(n) * 100.0 / gap;
            for (int k = 0; k < n; ++k)
                if (!(std::fabs(v[k] - z[(size_t)k * n]) <= tol)) return std::printf("z n=%d kind=%d k=%d\n", n, kind, k), 1;
        }
    // no memory: a status, no exception
    std::vector<double> d(500, 1.0), e(499, 0.3), v(500);
    double E = 0.0;
    for (size_t room : {(size_t)0, (size_t)5000, (size_t)200000}) {
        g_limit = g_held + room;
        const int rc = mcpi::tridiag_lowest(500, d.data(), e.data(), &E, v.data());
        g_limit = (size_t)-1;
        if (rc != -2) return std::printf("room %zu: status %d\n", room, rc), 1;
        d.assign(500, 1.0);
    }
    std::printf("ok\n");
    return 0;
}

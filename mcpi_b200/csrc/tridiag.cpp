// Symmetric tridiagonal eigensolver for the Lanczos matrix.
//
// The reference diagonalises the Lanczos tridiagonal with MKL's
// LAPACKE_dstev('V') (groundStateLieb.c:428-440). This is an own
// implementation of the implicit QL algorithm with Wilkinson shifts
// (Bowdler, Martin, Reinsch & Wilkinson, Numer. Math. 11 (1968) 293-306),
// accumulating the plane rotations into the eigenvector matrix, followed by an
// ascending sort. Contract as LAPACKE_dstev(ROW_MAJOR, 'V'): on return d holds
// the eigenvalues ascending and z[k*n + j] is component k of eigenvector j.
#include <algorithm>
#include <cmath>
#include <limits>
#include <memory>
#include <new>
#include <numeric>
#include <vector>

namespace mcpi {

namespace {

// Implicit QL: d becomes the eigenvalues (unsorted), e is destroyed; every
// plane rotation is handed to rot(i, c, s) in order, so that the eigenvector
// matrix is the product Z = G_1 G_2 ... of the rotations
// (z_i, z_i+1) <- (c z_i - s z_i+1, s z_i + c z_i+1) of its columns.
template <class Rot>
int ql(int n, double *d, double *e, Rot rot)
{
    const double eps = std::numeric_limits<double>::epsilon();
    for (int l = 0; l < n; ++l) {
        int iter = 0;
        for (;;) {
            int m = l;
            for (; m < n - 1; ++m) {
                const double dd = std::fabs(d[m]) + std::fabs(d[m + 1]);
                if (std::fabs(e[m]) <= eps * dd) break;
            }
            if (m == l) break;
            if (++iter > 64) return -1;
            // Wilkinson-type shift from the leading 2x2 block
            double g = (d[l + 1] - d[l]) / (2.0 * e[l]);
            double r = std::hypot(g, 1.0);
            g = d[m] - d[l] + e[l] / (g + (g >= 0 ? r : -r));
            double s = 1.0, c = 1.0, p = 0.0;
            int i = m - 1;
            bool deflated = false;
            for (; i >= l; --i) {
                const double f = s * e[i], b = c * e[i];
                r = std::hypot(f, g);
                e[i + 1] = r;
                if (r == 0.0) {  // underflow: split the matrix here
                    d[i + 1] -= p;
                    e[m] = 0.0;
                    deflated = true;
                    break;
                }
                s = f / r;
                c = g / r;
                g = d[i + 1] - p;
                r = (d[i] - g) * s + 2.0 * c * b;
                p = s * r;
                d[i + 1] = g + p;
                g = c * r - b;
                rot(i, c, s);
            }
            if (deflated) continue;
            d[l] -= p;
            e[l] = g;
            e[m] = 0.0;
        }
    }
    return 0;
}

}  // namespace

int tridiag_eig(int n, double *d, const double *e_in, double *z)
{
    if (n <= 0) return 0;
    std::vector<double> e(n, 0.0);
    for (int i = 0; i + 1 < n; ++i) e[i] = e_in[i];
    std::vector<double> Z;
    int rc;
    if (z) {
        Z.assign((size_t)n * n, 0.0);
        for (int i = 0; i < n; ++i) Z[(size_t)i * n + i] = 1.0;
        rc = ql(n, d, e.data(), [&](int i, double c, double s) {
            for (int k = 0; k < n; ++k) {
                double *zk = &Z[(size_t)k * n];
                const double fz = zk[i + 1];
                zk[i + 1] = s * zk[i] + c * fz;
                zk[i] = c * zk[i] - s * fz;
            }
        });
    } else {
        rc = ql(n, d, e.data(), [](int, double, double) {});
    }
    if (rc) return rc;
    std::vector<int> perm(n);
    std::iota(perm.begin(), perm.end(), 0);
    std::stable_sort(perm.begin(), perm.end(), [&](int a, int b) { return d[a] < d[b]; });
    std::vector<double> ds(d, d + n);
    for (int j = 0; j < n; ++j) d[j] = ds[perm[j]];
    if (z)
        for (int k = 0; k < n; ++k)
            for (int j = 0; j < n; ++j) z[(size_t)k * n + j] = Z[(size_t)k * n + perm[j]];
    return 0;
}

// The plane rotations of a QL run, read back in reverse order. Their indices
// fall by one within a sweep, so a rotation is its (c, s) and a sweep the index it
// starts with; blocks as they fill, so that nothing is held twice. A Lanczos
// matrix takes about n^2 rotations: 16 n^2 bytes, what tridiag_eig holds.
class Rotations {
    static constexpr size_t kBlock = 1024;
    struct CS {
        double c, s;
    };
    struct Sweep {
        int first;
        size_t at;
    };
    std::vector<std::unique_ptr<CS[]>> blocks_;
    std::vector<Sweep> sweeps_;
    size_t count_ = 0;
    int last_ = -1;

public:
    void add(int i, double c, double s)
    {
        if (sweeps_.empty() || i != last_ - 1) sweeps_.push_back({i, count_});
        if (count_ % kBlock == 0) blocks_.emplace_back(new CS[kBlock]);
        blocks_.back()[count_++ % kBlock] = {c, s};
        last_ = i;
    }
    template <class F>
    void reversed(F f) const
    {
        size_t x = count_;
        for (auto w = sweeps_.rbegin(); w != sweeps_.rend(); ++w)
            while (x > w->at) {
                --x;
                const CS &r = blocks_[x / kBlock][x % kBlock];
                f(w->first - (int)(x - w->at), r.c, r.s);
            }
    }
};

// The lowest eigenvalue of the tridiagonal (d, e) and its eigenvector z[n]: the
// same rotations as tridiag_eig, kept and applied backwards to the one unit
// vector whose column of Z is wanted -- O(n^2) instead of O(n^3) (n = 375: 8
// against 116 ms on one host core), the sign included. Ties take the first, as
// the ascending stable sort does. d is destroyed. -1: no convergence, -2: no
// host memory.
int tridiag_lowest(int n, double *d, const double *e_in, double *E, double *z)
try {
    if (n <= 0) return -1;
    std::vector<double> e(n, 0.0);
    for (int i = 0; i + 1 < n; ++i) e[i] = e_in[i];
    Rotations g;
    if (ql(n, d, e.data(), [&](int i, double c, double s) { g.add(i, c, s); })) return -1;
    int j = 0;
    for (int k = 1; k < n; ++k)
        if (d[k] < d[j]) j = k;
    *E = d[j];
    for (int k = 0; k < n; ++k) z[k] = k == j ? 1.0 : 0.0;
    g.reversed([&](int i, double c, double s) {
        const double a = z[i], b = z[i + 1];
        z[i] = c * a + s * b;
        z[i + 1] = c * b - s * a;
    });
    return 0;
} catch (const std::bad_alloc &) {
    return -2;
}

}  // namespace mcpi

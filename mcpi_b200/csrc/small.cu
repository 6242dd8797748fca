// Lanczos of a small space in one persistent launch.
//
// The launch sequence of lanczos.cu takes eight kernels per step. On a space of
// a few thousand configurations they leave the chip idle: at N=5, M=11 (3,003
// rows) 12 blocks do the update, each thread a serial chain over up to 375 basis
// vectors, and a step's 34 us are mostly launches and latency. Here the whole
// solve is one cooperative launch over all SMs with three grid barriers per step:
//   1. v_{i+1} = r / beta (whole, in every block's shared memory), and by rows
//      w = H v_{i+1} - beta v_i with the shares of alpha;
//   2. x = w - alpha v_{i+1} (whole, in shared memory), and one warp per
//      (basis vector, 1,024-row slice) the shares of <V_j, x>;
//   3. by rows r = x - sum_j c_j V_j: sixteen warps form the products of 64
//      vectors at a time, one subtracts them in order.
// Every sum is taken in the order of the launch sequence (lanczos.cu: 32-row
// warp sums, 256-row blocks, 1,024-row slices, vectors subtracted one by one)
// and every row of H.psi in that of the direct kernel (hpsi.cu: direct_row),
// so alpha, beta and the basis are bit for bit the launch sequence's
// (tests/test_gpu_small_lanczos.py). That is not for its own sake: with an
// odd number of plane waves the recurrence amplifies the last bit to order
// one and the Ritz vector's sign with it.
//
// H is applied from a stored list: the occupied creation pairs of a row (its
// groups), each with the coefficients and columns of its block's terms, built
// once at the start of each solve and read from L2 (a few MB).
//
// Measured (B200, N=5, M=11, 375 steps, whole mcpi_ground, of which 6.5 ms are the
// host's tridiagonal): 19.8 -> 12.8 ms.
// Barrier waits are bounded (about two seconds, then the status word reports
// MCPI_ERR_TIMEOUT and every block leaves at its next barrier).
#include <cuda_runtime.h>
#include "fock.cuh"
#include "kernels.h"
#include "mbarrier.cuh"

namespace mcpi {

namespace {

constexpr int kST = 512;          // threads per block
constexpr int kSW = kST / 32;     // warps per block
constexpr int kBuildT = 64;       // rows per block of the list builder
constexpr int kSliceS = 1024;     // rows of a dot product's share (lanczos.cu: kSlice)
constexpr int kChunk = 64;        // basis vectors whose products are staged together in the update

// The vector arithmetic of lanczos.cu with its fused multiply-adds written out
// (what the compiler makes of the plain expressions there; the test compares
// the results bit for bit, so a compiler that fuses otherwise shows there).
__device__ __forceinline__ double2 dot_term(double2 a, double2 b)   // conj(a) b
{
    return make_double2(__fma_rn(a.x, b.x, __dmul_rn(a.y, b.y)), __fma_rn(a.x, b.y, -__dmul_rn(a.y, b.x)));
}

__device__ __forceinline__ double2 prod(double2 p, double2 c)   // p c, to be subtracted
{
    return make_double2(__fma_rn(p.x, c.x, -__dmul_rn(p.y, c.y)), __fma_rn(p.y, c.x, __dmul_rn(p.x, c.y)));
}

__device__ __forceinline__ double2 warp_sum(double2 v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_down_sync(0xffffffffu, v.x, o);
        v.y += __shfl_down_sync(0xffffffffu, v.y, o);
    }
    return v;
}

// The rows of H as direct_row sums them: acc = h1 psi_i; the single-pair blocks
// before the others (acc += one[x] psi_i); per group acc += ca e with e the sum
// of its NB = M / 2 + 1 terms t psi_j in block order (shorter blocks end in
// zeros); the single-pair blocks after. Slices of 32 rows; group g of slice s
// has ca at (s cap + g) 32 + lane and term c at ((s cap + g) NB + c) 32 + lane.
struct RowLists {
    int cap, nb;
    int *groups;       // per slice: the longest row's
    double *ca, *t;
    uint32_t *col;
    double *h1;        // per row
    double *one;       // 5 per row (row-major by slice: x * 32 + lane): two before, three after
};

__global__ void __launch_bounds__(kBuildT) k_small_build(Space sp, SpaceTables tb, const double2 *__restrict__ hblk,
                                                       const double2 *__restrict__ hdiag, RowLists rl)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int M = sp.M, ws = sp.wstride, t = threadIdx.x;
    uint32_t *F = reinterpret_cast<uint32_t *>(smem_raw);   // M x kBuildT
    uint32_t *G = F + M * kBuildT;                          // M x kBuildT
    int *V = reinterpret_cast<int *>(G + M * kBuildT);      // M x kBuildT
    const uint32_t i = blockIdx.x * kBuildT + t;
    const bool row = i < sp.nc;
    const size_t slice = i / 32, lane = i % 32;
    const double *sq = tb.sq;
    int n = 0;
    if (row) {
        uint32_t R = sp.nc - 1u - i;
        int hi = sp.N;   // prefix counts from the top (fock.cuh: decode)
        V[(M - 1) * kBuildT + t] = sp.N;
        for (int o = M - 2; o >= 0; --o) {
            int p = hi;
            while (p > 0 && tb.W[o * ws + p] > R) --p;
            R -= tb.W[o * ws + p];
            V[o * kBuildT + t] = hi = p;
        }
        uint32_t f = 0, g = 0, s0 = 0;
        F[t] = G[t] = 0;
        for (int o = 1; o < M; ++o) {
            const int p = V[(o - 1) * kBuildT + t];
            const uint32_t w0 = tb.W[(o - 1) * ws + p];
            s0 += w0;
            f += tb.W[(o - 1) * ws + p + 1] - w0;
            g += (p > 0 ? tb.W[(o - 1) * ws + p - 1] : 0u) - w0;
            F[o * kBuildT + t] = f;
            G[o * kBuildT + t] = g;
        }
        for (int o = M - 1; o > 0; --o) V[o * kBuildT + t] -= V[(o - 1) * kBuildT + t];
        const uint32_t base = sp.nc - 1u - s0;
        double h1 = 0.0;
        for (int k = 0; k < M; ++k) h1 = __fma_rn(hdiag[k].x, (double)V[k * kBuildT + t], h1);
        rl.h1[i] = h1;
        for (int x = 0; x < 5; ++x) rl.one[(slice * 5 + x) * 32 + lane] = 0.0;
        int off = 0, after = 2;
        for (int K = 0; K <= 2 * M - 2; ++K) {
            const int qlo = K - (M - 1) > 0 ? K - (M - 1) : 0, nb = K / 2 - qlo + 1;
            if (nb == 1) {
                const int k = qlo, s = K - k, vk = V[k * kBuildT + t], vs = V[s * kBuildT + t];
                const double ca2 = k == s ? (double)(vk * (vk - 1)) : (double)(vk * vs);
                rl.one[(slice * 5 + (K < 2 ? K : after++)) * 32 + lane] = hblk[off].x * ca2;
                off += 1;
                continue;
            }
            for (int r = 0; r < nb; ++r) {
                const int k = qlo + r, s = K - k;
                const int vk = V[k * kBuildT + t], vs = V[s * kBuildT + t];
                if (k == s ? vk < 2 : (vk < 1 || vs < 1)) continue;
                const double ca = sq[vk] * sq[k == s ? vk - 1 : vs];
                const uint32_t XA = base - (F[k * kBuildT + t] - G[s * kBuildT + t]);
                const uint32_t XB = base - (F[s * kBuildT + t] - G[k * kBuildT + t]);
                rl.ca[(slice * rl.cap + n) * 32 + lane] = ca;
                for (int c = 0; c < rl.nb; ++c) {
                    double h = 0.0;
                    uint32_t j = i;
                    if (c < nb) {
                        const int q = qlo + c, l = K - q;
                        const int vq = V[q * kBuildT + t], vl = V[l * kBuildT + t];
                        const double w = c == r ? ca : sq[vq + 1] * sq[q == l ? vq + 2 : vl + 1];
                        h = hblk[off + r * nb + c].x * w;
                        if (c < r) j = XA + (F[q * kBuildT + t] - G[l * kBuildT + t]);
                        if (c > r) j = XB + (F[l * kBuildT + t] - G[q * kBuildT + t]);
                    }
                    const size_t at = ((slice * rl.cap + n) * rl.nb + c) * 32 + lane;
                    rl.t[at] = h;
                    rl.col[at] = j;
                }
                ++n;
            }
            off += nb * nb;
        }
    }
    // groups of the slice: the longest row's; shorter rows end in groups of zeros
    int most = n;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
    for (int g = n; g < most; ++g) {
        rl.ca[(slice * rl.cap + g) * 32 + lane] = 0.0;
        for (int c = 0; c < rl.nb; ++c) {
            const size_t at = ((slice * rl.cap + g) * rl.nb + c) * 32 + lane;
            rl.t[at] = 0.0;
            rl.col[at] = row ? i : 0u;
        }
    }
    if (lane == 0 && row) rl.groups[slice] = most;
}

struct SmallArgs {
    uint32_t nc;
    int lm;
    double tol;
    RowLists rl;
    double2 *V, *r, *w;       // basis (lm x nc); residual and H.psi, nc each
    double2 *alpha;           // lm
    double *beta;             // lm
    double2 *dotp, *part;     // shares: alpha per 32 rows; <V_j, x> per (j, slice)
    double *normp;            // shares: |r|^2 per 32 rows
    int *iters;
    unsigned *ctl;            // barrier counter, abort flag (zero at launch)
    int *status;
    long long wait_cycles;
    int test_stall;           // block 0 never arrives, so that the waits run out
};

// Grid barrier number k (0, 1, ..): false once any block has given up.
__device__ __forceinline__ bool grid_barrier(const SmallArgs &a, unsigned k)
{
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned want = (k + 1) * gridDim.x;
        const long long limit = a.wait_cycles > 0 ? a.wait_cycles : kWaitCycles;
        unsigned seen;
        int ok = 1;
        __threadfence();
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;\n" ::"l"(a.ctl) : "memory");
        const long long t0 = clock64();
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(seen) : "l"(a.ctl) : "memory");
            if (seen >= want) break;
            if (*(volatile unsigned *)(a.ctl + 32)) {
                ok = 0;
                break;
            }
            if (clock64() - t0 > limit) {
                atomicExch(a.ctl + 32, 1u);
                if (a.status) atomicExch(a.status, 1);
                ok = 0;
                break;
            }
        }
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// Sum of 32-row shares in the order of the launch sequence: eight shares to a
// 256-row block, thread b < 256 of the final sum takes block b, its warps are
// added in order (kSmallMaxRows: 22 blocks). One warp; the result is in lane 0.
template <class Load>
__device__ __forceinline__ double2 sum_shares(uint32_t nshares, Load load)
{
    const int lane = threadIdx.x % 32;
    double2 total = make_double2(0.0, 0.0);
    for (uint32_t b0 = 0; b0 * 8 < nshares; b0 += 32) {
        const uint32_t first = (b0 + lane) * 8;
        double2 x[8], s = make_double2(0.0, 0.0);
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = first + k < nshares ? load(first + k) : make_double2(0.0, 0.0);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            s.x += x[k].x;
            s.y += x[k].y;
        }
        s = warp_sum(s);
        total.x += s.x;
        total.y += s.y;
    }
    return total;
}

__global__ void __launch_bounds__(kST, 1) k_small_lanczos(SmallArgs a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2 *xs = reinterpret_cast<double2 *>(smem_raw);   // nc: v_{i+1}, then x
    double2 *cs = xs + a.nc;                               // lm coefficients
    double2 *ex = cs + a.lm;                               // a tile's group sums, or a chunk's products
    __shared__ double2 s_val;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const uint32_t nc = a.nc, ntiles = (nc + 31) / 32;
    const int nslices = (int)((nc + kSliceS - 1) / kSliceS);
    const RowLists &rl = a.rl;
    unsigned nbar = 0;
    double beta = 0.0, maxbeta = 0.0;
    if (a.test_stall && blockIdx.x == 0) return;
    for (int i = -1; i < a.lm - 1; ++i) {
        // this step makes v_{i+1} (i = -1: v_0 is given), alpha_{i+1} and the next residual
        double2 *vn = a.V + (size_t)(i + 1) * nc;
        if (i >= 0) {
            if (warp == 0) {
                const double2 s =
                    sum_shares(ntiles, [&](uint32_t x) { return make_double2(__ldcg(a.normp + x), 0.0); });
                if (lane == 0) s_val.x = sqrt(s.x);
            }
            __syncthreads();
            beta = s_val.x;
            if (maxbeta < beta) maxbeta = beta;
            if (blockIdx.x == 0 && threadIdx.x == 0) a.beta[i] = beta;
            if (!(beta / maxbeta >= a.tol)) {   // breakdown (groundStateLieb.c:287-292), the same in every block
                if (blockIdx.x == 0 && threadIdx.x == 0) *a.iters = i;
                return;
            }
            for (uint32_t x = threadIdx.x; x < nc; x += kST) {
                const double2 y = __ldcg(a.r + x);
                xs[x] = make_double2(y.x / beta, y.y / beta);
            }
        } else {
            for (uint32_t x = threadIdx.x; x < nc; x += kST) xs[x] = __ldcg(vn + x);
        }
        __syncthreads();
        // 1. rows: w = H v_{i+1} - beta v_i, shares of <v_{i+1}, w>
        for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
            const uint32_t row = tile * 32 + lane;
            const int ng = rl.groups[tile];
            const size_t g0 = (size_t)tile * rl.cap;
            for (int g = warp; g < ng; g += kSW) {
                double2 e = make_double2(0.0, 0.0);
                const size_t at = (g0 + g) * rl.nb * 32 + lane;
#pragma unroll 6
                for (int c = 0; c < rl.nb; ++c) {
                    const double h = rl.t[at + c * 32];
                    const double2 y = xs[rl.col[at + c * 32]];
                    e.x = fma(h, y.x, e.x);
                    e.y = fma(h, y.y, e.y);
                }
                ex[g * 32 + lane] = e;
            }
            __syncthreads();
            if (warp == 0) {
                double2 d = make_double2(0.0, 0.0);
                if (row < nc) {
                    const double2 x0 = xs[row];
                    const double h1 = rl.h1[row];   // Ho's diagonal is real here
                    double2 acc = make_double2(__dmul_rn(h1, x0.x), __dmul_rn(h1, x0.y));
                    const double *one = rl.one + (size_t)tile * 5 * 32 + lane;
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        acc.x = fma(one[x * 32], x0.x, acc.x);
                        acc.y = fma(one[x * 32], x0.y, acc.y);
                    }
                    for (int g = 0; g < ng; ++g) {
                        const double ca = rl.ca[(g0 + g) * 32 + lane];
                        const double2 e = ex[g * 32 + lane];
                        acc.x = fma(ca, e.x, acc.x);
                        acc.y = fma(ca, e.y, acc.y);
                    }
#pragma unroll
                    for (int x = 2; x < 5; ++x) {
                        acc.x = fma(one[x * 32], x0.x, acc.x);
                        acc.y = fma(one[x * 32], x0.y, acc.y);
                    }
                    double2 y = acc;
                    if (i >= 0) {
                        const double2 p = __ldcg(a.V + (size_t)i * nc + row);
                        y.x = __fma_rn(-beta, p.x, y.x);
                        y.y = __fma_rn(-beta, p.y, y.y);
                        vn[row] = x0;
                    }
                    a.w[row] = y;
                    d = dot_term(x0, y);
                }
                d = warp_sum(d);
                if (lane == 0) a.dotp[tile] = d;
            }
            __syncthreads();
        }
        if (!grid_barrier(a, nbar++)) return;
        // 2. alpha, x = w - alpha v_{i+1}, shares of <V_j, x>
        if (warp == 0) {
            const double2 s = sum_shares(ntiles, [&](uint32_t x) { return __ldcg(a.dotp + x); });
            if (lane == 0) s_val = s;
        }
        __syncthreads();
        const double2 al = s_val;
        if (blockIdx.x == 0 && threadIdx.x == 0) a.alpha[i + 1] = al;
        if (i + 1 >= a.lm - 1) return;   // the last alpha needs no residual
        for (uint32_t x = threadIdx.x; x < nc; x += kST) {
            const double2 y = __ldcg(a.w + x), t = prod(al, xs[x]);
            xs[x] = make_double2(y.x - t.x, y.y - t.y);
        }
        __syncthreads();
        const int nvec = i < 0 ? 0 : i + 2;
        for (int task = warp * gridDim.x + blockIdx.x; task < nvec * nslices; task += kSW * gridDim.x) {
            const int j = task / nslices, s = task % nslices;
            const uint32_t r0 = s * kSliceS;
            const int rows = (int)(nc - r0 < kSliceS ? nc - r0 : kSliceS);
            const double2 *vj = a.V + (size_t)j * nc + r0;
            double2 acc = make_double2(0.0, 0.0);
#pragma unroll 8
            for (int t = lane; t < rows; t += 32) {
                const double2 p = dot_term(__ldcg(vj + t), xs[r0 + t]);
                acc.x += p.x;
                acc.y += p.y;
            }
            acc = warp_sum(acc);
            if (lane == 0) a.part[(size_t)j * nslices + s] = acc;
        }
        if (nvec && !grid_barrier(a, nbar++)) return;
        // 3. rows: r = x - sum_j c_j V_j, shares of |r|^2
        for (int j = threadIdx.x; j < nvec; j += kST) {
            // the warp sum of k_multidot_finish over the slices (six at most)
            double2 p[16];
#pragma unroll
            for (int s = 0; s < 16; ++s)
                p[s] = s < nslices ? __ldcg(a.part + (size_t)j * nslices + s) : make_double2(0.0, 0.0);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1)
#pragma unroll
                for (int s = 0; s < o; ++s) {
                    p[s].x += p[s + o].x;
                    p[s].y += p[s + o].y;
                }
            cs[j] = p[0];
        }
        __syncthreads();
        for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
            const uint32_t row = tile * 32 + lane;
            constexpr int kPer = kChunk / kSW;   // vectors of a chunk per warp
            double2 p[kPer], u = make_double2(0.0, 0.0);
            if (row < nc) u = xs[row];
            auto fetch = [&](int j0) {
#pragma unroll
                for (int q = 0; q < kPer; ++q) {
                    const int j = j0 + warp * kPer + q;
                    p[q] = j < nvec && row < nc ? __ldcg(a.V + (size_t)j * nc + row) : make_double2(0.0, 0.0);
                }
            };
            fetch(0);
            for (int j0 = 0; j0 < nvec; j0 += kChunk) {
#pragma unroll
                for (int q = 0; q < kPer; ++q) {
                    const int j = j0 + warp * kPer + q;
                    const double2 c = j < nvec ? cs[j] : make_double2(0.0, 0.0);
                    ex[(warp * kPer + q) * 32 + lane] = prod(p[q], c);
                }
                __syncthreads();
                fetch(j0 + kChunk);
                if (warp == 0) {
                    const int n = nvec - j0 < kChunk ? nvec - j0 : kChunk;
#pragma unroll 8
                    for (int q = 0; q < n; ++q) {
                        const double2 t = ex[q * 32 + lane];
                        u.x -= t.x;
                        u.y -= t.y;
                    }
                }
                __syncthreads();
            }
            if (warp == 0) {
                double2 nn = make_double2(0.0, 0.0);
                if (row < nc) {
                    a.r[row] = u;
                    nn.x = __fma_rn(u.y, u.y, __dmul_rn(u.x, u.x));
                }
                nn = warp_sum(nn);
                if (lane == 0) a.normp[tile] = nn.x;
            }
        }
        if (!grid_barrier(a, nbar++)) return;
    }
}

size_t up(size_t x) { return (x + 255) & ~size_t(255); }

// Most creation pairs that a row of N particles holds.
int group_cap(const Space &sp)
{
    const int P = sp.M * (sp.M + 1) / 2;
    const long long held = (long long)sp.N * (sp.N - 1) / 2 + sp.N / 2;
    return (int)(held < P ? held : P);
}

// Dynamic shared memory of the solve.
size_t small_smem(const Space &sp, int lm)
{
    const int cap = group_cap(sp);
    return sizeof(double2) * ((size_t)sp.nc + lm + 32 * (size_t)(cap > kChunk ? cap : kChunk));
}

// Workspace: one block, the parts below in order.
struct SmallLayout {
    size_t groups, ca, t, col, h1, one, w, dotp, part, normp, ctl, bytes;
    SmallLayout(const Space &sp, int lm)
    {
        const size_t slices = (sp.nc + 31) / 32, rows = slices * 32, cap = group_cap(sp), nb = sp.M / 2 + 1;
        size_t at = 0;
        auto take = [&](size_t b) {
            const size_t o = at;
            at += up(b);
            return o;
        };
        groups = take(sizeof(int) * slices);
        ca = take(sizeof(double) * rows * cap);
        t = take(sizeof(double) * rows * cap * nb);
        col = take(sizeof(uint32_t) * rows * cap * nb);
        h1 = take(sizeof(double) * rows);
        one = take(sizeof(double) * rows * 5);
        w = take(sizeof(double2) * sp.nc);
        dotp = take(sizeof(double2) * slices);
        part = take(sizeof(double2) * lm * ((sp.nc + kSliceS - 1) / kSliceS));
        normp = take(sizeof(double) * slices);
        ctl = take(sizeof(unsigned) * 64);
        bytes = at;
    }
};

// The solves that it takes: up to this many rows (every block keeps the whole
// vector in shared memory and reads it twice a step, which grows with the rows
// while the launch sequence's short kernels do not), and enough steps to pay for
// the lists, one per 128 rows. mcpi_ground in ms, one launch / launch sequence:
//   N=18, M=4 (1,330 rows) 8 steps 0.20 / 0.28, 500 steps 17.6 / 25.2;
//   N=5, M=11 (3,003) 40 steps 0.87 / 1.23, 500 steps 19.1 / 29.0;
//   N=10, M=6 (3,003) 8 steps 0.239 / 0.232, 40 steps 0.85 / 0.99;
//   N=9, M=7 (5,005) 8 steps 0.264 / 0.244, 40 steps 1.01 / 1.05, 500 steps 23.6 / 26.7;
//   N=12, M=6 (6,188) 100 steps 2.78 / 2.70, 500 steps 24.6 / 26.2;
//   N=14, M=6 (11,628) 100 steps 3.90 / 2.69.
constexpr uint32_t kSmallMaxRows = 5500;
constexpr int kSmallMinSteps = 8, kSmallMaxSteps = 2048;
constexpr uint32_t kSmallRowsPerStep = 128;
// Its shared memory never exceeds that of the largest such solve (66 pairs: M = 11).
constexpr size_t kSmallSmem = sizeof(double2) * (kSmallMaxRows + kSmallMaxSteps + 32 * 66);
static_assert(kSmallSmem <= 226 * 1024 && kDirectAutoMaxM * (kDirectAutoMaxM + 1) / 2 == 66 && kChunk <= 66,
              "a block may have 227 KB, 1 KB of it static");

}  // namespace

bool small_lanczos_fits(const Space &sp, int lm)
{
    return sp.M >= 2 && sp.N >= 2 && direct_covers(sp) && sp.nc <= kSmallMaxRows && lm >= kSmallMinSteps &&
           lm <= kSmallMaxSteps && kSmallRowsPerStep * (uint32_t)lm >= sp.nc;
}

size_t small_lanczos_bytes(const Space &sp, int lm) { return SmallLayout(sp, lm).bytes; }

cudaError_t launch_small_lanczos(const Space &sp, const SpaceTables &tb, const PairOp &op, double2 *V, int lm,
                                 double tol, double2 *r, LanczosState s, void *work, int device, cudaStream_t st)
{
    const SmallLayout lay(sp, lm);
    char *b = static_cast<char *>(work);
    SmallArgs a{};
    a.nc = sp.nc;
    a.lm = lm;
    a.tol = tol;
    a.rl.cap = group_cap(sp);
    a.rl.nb = sp.M / 2 + 1;
    a.rl.groups = reinterpret_cast<int *>(b + lay.groups);
    a.rl.ca = reinterpret_cast<double *>(b + lay.ca);
    a.rl.t = reinterpret_cast<double *>(b + lay.t);
    a.rl.col = reinterpret_cast<uint32_t *>(b + lay.col);
    a.rl.h1 = reinterpret_cast<double *>(b + lay.h1);
    a.rl.one = reinterpret_cast<double *>(b + lay.one);
    a.V = V;
    a.r = r;
    a.w = reinterpret_cast<double2 *>(b + lay.w);
    a.alpha = s.alpha;
    a.beta = s.beta;
    a.dotp = reinterpret_cast<double2 *>(b + lay.dotp);
    a.part = reinterpret_cast<double2 *>(b + lay.part);
    a.normp = reinterpret_cast<double *>(b + lay.normp);
    a.iters = s.iters;
    a.ctl = reinterpret_cast<unsigned *>(b + lay.ctl);
    a.status = op.status;
    a.wait_cycles = op.wait_cycles;
    a.test_stall = op.test_stall;
    int sms = 0, per = 0;
    const size_t sm = small_smem(sp, lm);
    const void *fn = (const void *)k_small_lanczos;
    cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallSmem);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, kST, sm);
    if (e != cudaSuccess) return e;
    if (per < 1) return cudaErrorCooperativeLaunchTooLarge;   // the caller runs the launch sequence
    if ((e = cudaMemsetAsync(a.ctl, 0, sizeof(unsigned) * 64, st)) != cudaSuccess) return e;
    k_small_build<<<(sp.nc + kBuildT - 1) / kBuildT, kBuildT, 3 * sizeof(uint32_t) * sp.M * kBuildT, st>>>(
        sp, tb, op.hblk, op.hdiag, a.rl);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    void *args[] = {&a};
    return cudaLaunchCooperativeKernel(fn, dim3(sms), dim3(kST), args, sm, st);
}

}  // namespace mcpi

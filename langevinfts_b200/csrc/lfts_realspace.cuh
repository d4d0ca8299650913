// Real-space Crank-Nicolson step for continuous chains (the reference's
// "realspace" method, src/platforms/cpu/CpuSolverReal.cpp:135-549 and
// src/platforms/cuda/CudaSolverReal.cu:371-956): for boxes with reflecting or
// absorbing walls, where the pseudo-spectral step does not apply.
//
//   q_out = e * ADI(e * q_in),  e = exp(-w ds / 2)
//
// ADI (alternating direction implicit, the reference's scheme): a first sweep
// implicit along the box's first axis whose right-hand side applies the full
// explicit half of the operator, then one sweep per further axis implicit
// along it, each a batch of independent tridiagonal solves (periodic axes by
// Sherman-Morrison).  The pivots of every axis depend only on its matrix, so
// the host computes them once (lfts_realspace_tables) and a line solve is the
// reference's forward and backward substitution with those pivots.
//
// Launch shape: a block takes W neighbouring lines of one axis (blockIdx.y =
// job).  All its threads compute right-hand sides into a shared-memory tile,
// with accesses to global memory in its order whatever the axis (rows of W + 1
// doubles keep both orders off each other's banks), one warp then solves, a line
// a lane, and all threads write the tile back.  The substitutions are one chain each,
// whose operands come from shared memory ahead of it: a fused multiply-add and the
// product with the reciprocal pivot an element (folding that into the right-hand
// sides and the off-diagonals takes one operation off the chain, 2 % of a film's
// step, but rounds a matrix entry that every step applies again: 200 points, 100
// steps 5.2e-15 off instead of 3.6e-15).  One thread a line straight from global
// memory left 24 CTAs waiting on every element: 72 us a sweep at 48 x 48 x 64, 2 jobs.
#pragma once
#include "lfts_step_kernels.cuh"

namespace lfts {
namespace rs {

constexpr int ROWS = 7;  // l, d, h, pivot, ratio, periodic vector, 1 / pivot

// view of one type's tables (device doubles, layout of lfts_realspace_tables)
struct Axis {
    const double *l, *d, *h, *c, *v, *rp;
    double denom;
    bool periodic;
    int n;
};
__device__ __forceinline__ Axis axis(const double *tab, const GridPlan &g, int a) {
    const int n[3] = {g.n0, g.n1, g.n2};
    long long off = 0;
    for (int b = 0; b < a; b++) off += (long long)ROWS * n[b];
    const double *t = tab + off;
    const long long tail = (long long)ROWS * (n[0] + n[1] + n[2]);
    Axis ax;
    ax.n = n[a];
    ax.l = t;
    ax.d = t + n[a];
    ax.h = t + 2 * n[a];
    ax.c = t + 4 * n[a];
    ax.v = t + 5 * n[a];
    ax.rp = t + 6 * n[a];
    ax.denom = tab[tail + a];
    ax.periodic = tab[tail + 3 + a] != 0.0;
    return ax;
}
__device__ __forceinline__ int nb_lo(const Axis &ax, int i) { return i > 0 ? i - 1 : ax.periodic ? ax.n - 1 : 0; }
__device__ __forceinline__ int nb_hi(const Axis &ax, int i) { return i < ax.n - 1 ? i + 1 : ax.periodic ? 0 : ax.n - 1; }

// e * q at flat index m (e = fac^2)
__device__ __forceinline__ double eq(const double *q, const double *fac, long long m) {
    const double f = fac[m];
    return q[m] * (f * f);
}

// shared memory of a block: the tile and six rows of the axis's tables
constexpr int T_ROWS = 6;  // l, d, h, 1 / pivot, ratio, periodic vector
__host__ __device__ constexpr size_t tile_smem(int n, int W) { return sizeof(double) * ((size_t)n * (W + 1) + T_ROWS * (size_t)n); }

// Flat index of element i of line `line` along padded axis A
template <int A> __device__ __forceinline__ int point(const GridPlan &g, int line, int i) {
    if (A == 0) return i * g.n1 * g.n2 + line;  // lines (j, k) -> j n2 + k
    if (A == 1) {
        const int x = line / g.n2;  // lines (i, k) -> i n2 + k
        return (x * g.n1 + i) * g.n2 + line - x * g.n2;
    }
    return line * g.n2 + i;  // lines (i, j) -> i n1 + j
}

// One sweep along padded axis A.  FIRST: the right-hand side is the explicit
// operator of all axes on e q (CpuSolverReal.cpp:223-242, 2D :355-373, 1D
// :437-449).  Otherwise prev + (d - 1) e q + l e q[-] + h e q[+] along A
// (:250-306, 2D :382-400).  LAST: the solution times e goes to q_out, else to the
// scratch half src_half does not name.
constexpr int NT = 512;
template <int DIM, int A, bool FIRST, bool LAST, int W>
__global__ void __launch_bounds__(NT) k_rs_sweep(GridPlan g, const lfts_step_job *__restrict__ jobs, int s, int src_half) {
    extern __shared__ double sm_rs[];
    grid_wait();  // before the job array too: FIRST is the first kernel of a step
    const lfts_step_job jb = jobs[blockIdx.y];
    if (jb.active && !jb.active[jb.replica]) return;
    constexpr int ld = W + 1;
    const double *q = (const double *)jb.in + s * jb.in_stride, *fac = (const double *)jb.fac, *tab = (const double *)jb.bond;
    const Axis X = axis(tab, g, A), Y = axis(tab, g, 1), Z = axis(tab, g, 2);
    const int st = A == 0 ? g.n1 * g.n2 : A == 1 ? g.n2 : 1;  // between neighbours along A
    const int n = X.n, nlines = (int)(g.M / n), line0 = blockIdx.x * W, nl = min(W, nlines - line0);
    double *tile = sm_rs, *tl = tile + n * ld, *td = tl + n, *th = td + n, *tp = th + n, *tc = tp + n, *tv = tc + n;
    for (int i = threadIdx.x; i < n; i += NT) {
        tl[i] = X.l[i];
        td[i] = X.d[i];
        th[i] = X.h[i];
        tp[i] = X.rp[i];
        tc[i] = X.c[i];
        tv[i] = X.v[i];
    }
    __syncthreads();
    const double *prev = (const double *)jb.spec + (src_half ? g.M : 0);
    double *dst = LAST ? (double *)jb.out + s * jb.out_stride : (double *)jb.spec + (FIRST || src_half ? 0 : g.M);
    // element t of the tile in the order of global memory: (line, i)
    auto element = [&](int t, int &w, int &i) {
        if (A == 2) {
            w = t / n;
            i = t - w * n;
        } else {
            i = t / W;
            w = t - i * W;
        }
    };
    const int tot = A == 2 ? nl * n : n * W;
#pragma unroll 4
    for (int t = threadIdx.x; t < tot; t += NT) {
        int w, i;
        element(t, w, i);
        const int line = min(line0 + w, nlines - 1), m = point<A>(g, line, i);  // a short block's spare columns repeat a line
        const double E = eq(q, fac, m), Em = eq(q, fac, m + (nb_lo(X, i) - i) * st), Ep = eq(q, fac, m + (nb_hi(X, i) - i) * st);
        double r;
        if (!FIRST) {
            r = prev[m] + (td[i] - 1.0) * E + tl[i] * Em + th[i] * Ep;
        } else if (DIM == 1) {
            r = (2.0 - td[i]) * E - tl[i] * Em - th[i] * Ep;
        } else {
            const int j = DIM == 2 ? 0 : line / g.n2, k = line - j * g.n2, km = nb_lo(Z, k) - k, kp = nb_hi(Z, k) - k;
            if (DIM == 2) {
                r = 2.0 * ((2.0 - 0.5 * td[i] - Z.d[k]) * E - Z.l[k] * eq(q, fac, m + km) - Z.h[k] * eq(q, fac, m + kp)) -
                    tl[i] * Em - th[i] * Ep;
            } else {
                const int jm = (nb_lo(Y, j) - j) * g.n2, jp = (nb_hi(Y, j) - j) * g.n2;
                r = 2.0 * ((3.0 - 0.5 * td[i] - Y.d[j] - Z.d[k]) * E - Z.l[k] * eq(q, fac, m + km) - Z.h[k] * eq(q, fac, m + kp) -
                           Y.l[j] * eq(q, fac, m + jm) - Y.h[j] * eq(q, fac, m + jp)) -
                    tl[i] * Em - th[i] * Ep;
            }
        }
        tile[i * ld + w] = r;
    }
    __syncthreads();
    if (threadIdx.x < nl) {
        double *x = tile + threadIdx.x, v = x[0] * tp[0];
        x[0] = v;
#pragma unroll 8
        for (int i = 1; i < n; i++) {
            v = (x[i * ld] - tl[i] * v) * tp[i];
            x[i * ld] = v;
        }
#pragma unroll 8
        for (int i = n - 2; i >= 0; i--) {
            v = x[i * ld] - tc[i] * v;
            x[i * ld] = v;
        }
    }
    __syncthreads();
#pragma unroll 4
    for (int t = threadIdx.x; t < tot; t += NT) {
        int w, i;
        element(t, w, i);
        if (w >= nl) continue;
        const int m = point<A>(g, line0 + w, i);
        double v = tile[i * ld + w];
        if (X.periodic) v -= tv[i] * ((tile[w] + tl[0] * tile[(n - 1) * ld + w]) / X.denom);
        if (LAST) {
            const double f = fac[m];
            v *= f * f;
        }
        dst[m] = v;
    }
}

}  // namespace rs
}  // namespace lfts

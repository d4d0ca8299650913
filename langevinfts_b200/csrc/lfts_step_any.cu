// Plans and launches of the any-extent step kernels (lfts_step_any.cuh).
#include "lfts_any.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "lfts_step_any.cuh"

namespace lfts {

struct AnyGrid {
    any::Plan p;
    int prec = 8, nsm = 148, max_smem = 0;
    int stress_smem = 0;  // dynamic shared memory left to ka_xstress by its static reduction scratch
    void *tables = nullptr;
    // clusters of 1, 2, 4, 8, 16 CTAs the device holds at once (0: no fit), asked of it at
    // creation, so that the rule below gives a grid and a number of jobs one size for good
    int clusters_cont[5] = {0, 0, 0, 0, 0}, clusters_disc[5] = {0, 0, 0, 0, 0};
};

namespace {
using any::Plan;

// Fewest stages first, then the smallest sum of radices, radices never rising from the
// outermost on: every product of the primes up to 13 has such an order, so a branch that
// its cap leaves without a radix is a dead end (an odd composite taken there as a prime
// made 98 a radix-49 pair sum instead of 7 x 7 x 2).
void best_radices(int n, std::vector<int> &cur, std::vector<int> &best, int most) {
    if (n == 1) {
        auto sum = [](const std::vector<int> &v) { int s = 0; for (int x : v) s += x; return s; };
        if (best.empty() || cur.size() < best.size() || (cur.size() == best.size() && sum(cur) < sum(best))) best = cur;
        return;
    }
    if (!best.empty() && cur.size() >= best.size()) return;
    static const int regs[] = {16, 13, 12, 11, 10, 9, 8, 7, 6, 5, 4, 3, 2};
    for (int r : regs)
        if (r <= most && n % r == 0) {
            cur.push_back(r);
            best_radices(n / r, cur, best, r);
            cur.pop_back();
        }
}

bool make_axis(int n, any::Axis &ax, std::vector<short> &perm, std::vector<short> &iperm) {
    std::vector<int> r;
    if (!any_radices(n, r)) return false;
    ax.n = n;
    ax.nf = (int)r.size();
    int span = n;
    for (int f = 0; f < ax.nf; f++) {
        span /= r[f];
        ax.st[f] = {r[f], span, any::div_mul(span), n / r[f], n / (span * r[f])};
    }
    perm.assign(n, 0);
    iperm.assign(n, 0);
    for (int t = 0; t < n; t++) {
        int pos = 0, len = n, rem = t;
        for (int f = 0; f < ax.nf; f++) {
            len /= r[f];
            pos += (rem % r[f]) * len;
            rem /= r[f];
        }
        perm[t] = (short)pos;
        iperm[pos] = (short)t;
    }
    return true;
}

// dynamic shared memory a kernel may have: the block's less its own static part
template <typename K> int dynamic_limit(K kernel, int max_smem) {
    cudaFuncAttributes fa;
    return cudaFuncGetAttributes(&fa, kernel) == cudaSuccess ? max_smem - (int)fa.sharedSizeBytes : 0;
}
template <typename K> bool allow(K kernel, int max_smem, bool cluster = false) {
    const int limit = dynamic_limit(kernel, max_smem);
    if (limit <= 0 || cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, limit) != cudaSuccess) return false;
    return !cluster || cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
}
template <typename T> bool allow_all(int max_smem) {
    return allow(any::ka_plane_forward<T, true>, max_smem) && allow(any::ka_plane_forward<T, false>, max_smem) &&
           allow(any::ka_plane_mid<T, false>, max_smem) && allow(any::ka_plane_mid<T, true>, max_smem) && allow(any::ka_plane_inverse<T, true>, max_smem) &&
           allow(any::ka_plane_inverse<T, false>, max_smem) && allow(any::ka_plane_seam<T>, max_smem) && allow(any::ka_xpass<T, 1>, max_smem) &&
           allow(any::ka_xpass<T, 2>, max_smem) && allow(any::ka_xpass_forward<T>, max_smem) && allow(any::ka_xstress<T>, max_smem) &&
           allow(any::ka_sweep_continuous<T>, max_smem, true) && allow(any::ka_sweep_discrete<T>, max_smem, true);
}

int ceil_div(int a, int b) { return (a + b - 1) / b; }

any::Stack stack(const Plan &g, int planes) { return {planes, any::div_mul(planes * g.n1), any::div_mul(planes * g.n2)}; }

struct SweepShape {
    any::Sweep w;
    size_t smem;
};
template <typename C> SweepShape sweep_shape(const Plan &g, bool continuous, int cs) {
    SweepShape s;
    any::Sweep &w = s.w;
    w.XB = ceil_div(g.n0, cs);
    w.JB = ceil_div(g.n1 * g.nzc, cs);
    w.width = continuous ? 2 * w.JB : w.JB;
    w.mul_xb = any::div_mul(w.XB);
    w.mul_jb = any::div_mul(w.JB);
    w.mul_width = any::div_mul(w.width);
    w.all = stack(g, w.XB);
    w.half = stack(g, (w.XB + 1) / 2);
    s.smem = any::SweepBuf<C>::bytes(g, continuous ? w.XB : w.half.planes, w.width);
    return s;
}
SweepShape sweep_shape(const AnyGrid *a, bool continuous, int cs) {
    return a->prec == 8 ? sweep_shape<double2>(a->p, continuous, cs) : sweep_shape<float2>(a->p, continuous, cs);
}
int sweep_threads(const AnyGrid *a, const SweepShape &s) {
    // a thread for every four points of the slab's packed planes
    const int want = s.w.XB * a->p.n1 * a->p.n2 / 4;
    return std::min(any::NT_MAX, std::max(128, (want + 31) / 32 * 32));
}

template <typename K> void cluster_config(cudaLaunchConfig_t &cfg, cudaLaunchAttribute *at, K, int cs, int nj, int threads, size_t smem,
                                          cudaStream_t st) {
    std::memset(&cfg, 0, sizeof cfg);
    cfg.gridDim = dim3(cs, nj);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = cs;
    at->val.clusterDim.y = 1;
    at->val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
}

template <typename K> int resident_clusters(const AnyGrid *a, K kernel, bool continuous, int cs) {
    const SweepShape s = sweep_shape(a, continuous, cs);
    if (s.smem > (size_t)a->max_smem) return 0;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at;
    cluster_config(cfg, &at, kernel, cs, 64, sweep_threads(a, s), s.smem, 0);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    return n;
}

template <typename T> bool setup(AnyGrid *a, std::string &err) {
    using C = typename CT<T>::type;
    Plan &g = a->p;
    std::vector<short> perm[3], iperm[3];
    for (int d = 0; d < 3; d++)
        if (!make_axis(d == 0 ? g.n0 : d == 1 ? g.n1 : g.n2, g.ax[d], perm[d], iperm[d])) return false;
    if (any::PlaneBuf<C>::bytes(g, 1) > (size_t)a->max_smem || any::TileBuf<C>::bytes(g, 2 * 4) > (size_t)a->max_smem) return false;
    size_t bytes = 0;
    for (int d = 0; d < 3; d++) bytes += (sizeof(C) * g.ax[d].n + 15) / 16 * 16 + 2 * ((sizeof(short) * g.ax[d].n + 15) / 16 * 16);
    std::vector<unsigned char> host(bytes, 0);
    if (cudaMalloc(&a->tables, bytes) != cudaSuccess) { err = "allocation of the transform tables failed"; return false; }
    size_t off = 0;
    for (int d = 0; d < 3; d++) {
        const int n = g.ax[d].n;
        C *tw = (C *)(host.data() + off);
        for (int j = 0; j < n; j++) {
            const long double ang = -2.0L * 3.141592653589793238462643383279502884L * (long double)j / (long double)n;
            tw[j].x = (T)std::cos(ang);
            tw[j].y = (T)std::sin(ang);
        }
        g.tw[d] = (const char *)a->tables + off;
        off += (sizeof(C) * n + 15) / 16 * 16;
        const std::vector<short> *tab[2] = {&perm[d], &iperm[d]};
        const short **dst[2] = {&g.perm[d], &g.iperm[d]};
        for (int k = 0; k < 2; k++) {
            std::memcpy(host.data() + off, tab[k]->data(), sizeof(short) * n);
            *dst[k] = (const short *)((const char *)a->tables + off);
            off += (sizeof(short) * n + 15) / 16 * 16;
        }
    }
    if (cudaMemcpy(a->tables, host.data(), bytes, cudaMemcpyHostToDevice) != cudaSuccess || !allow_all<T>(a->max_smem)) {
        err = std::string("transform setup: ") + cudaGetErrorString(cudaGetLastError());
        return false;
    }
    a->stress_smem = dynamic_limit(any::ka_xstress<T>, a->max_smem);
    for (int k = 0; k < 5; k++) {
        a->clusters_cont[k] = resident_clusters(a, any::ka_sweep_continuous<T>, true, 1 << k);
        a->clusters_disc[k] = resident_clusters(a, any::ka_sweep_discrete<T>, false, 1 << k);
    }
    return true;
}

// x-planes (or packed pairs) a plane CTA takes: small planes are stacked while
// the launch still has two CTAs for every SM
template <typename C> int stack_planes(const AnyGrid *a, int units, int nj) {
    const Plan &g = a->p;
    int k = 1;
    while (k * g.n1 * g.n2 < 2048 && (long long)ceil_div(units, 2 * k) * nj >= 2 * a->nsm &&
           any::PlaneBuf<C>::bytes(g, 2 * k) <= (size_t)a->max_smem / 2)
        k *= 2;
    return k;
}
int plane_threads(const AnyGrid *a, int ctas, int points) {
    const int most = ctas <= a->nsm ? any::NT_MAX : 256;
    return std::min(most, std::max(64, (points / 4 + 31) / 32 * 32));
}
// limit: dynamic shared memory of the kernel that takes the tile
template <typename C> int tile_columns(const AnyGrid *a, int nbr, int nj, int limit) {
    const Plan &g = a->p;
    int tj = sizeof(C) == 16 ? 16 : 32;
    const int cols = g.n1 * g.nzc;
    // narrower tiles (still whole 64-byte rows) when wide ones leave SMs without work or do not fit
    while (tj > 4 && (any::TileBuf<C>::bytes(g, nbr * tj) > (size_t)limit ||
                      ((long long)ceil_div(cols, tj) * nj < a->nsm && tj * sizeof(C) > 128)))
        tj /= 2;
    return tj;
}

// in_step: with the programmatic edge of the step kernels (the kernel reads the job array after its wait)
template <typename T, bool TWO> void plane_forward(const AnyGrid *a, cudaStream_t st, const lfts_step_job *jobs, int nj, int s, int f0, int f1, int spec, bool in_step = true) {
    using C = typename CT<T>::type;
    const Plan &g = a->p;
    const int units = TWO ? g.n0 : ceil_div(g.n0, 2), k = stack_planes<C>(a, units, nj), ctas = ceil_div(units, k);
    const dim3 grid(ctas, nj);
    const int threads = plane_threads(a, ctas * nj, k * g.n1 * g.n2);
    const size_t smem = any::PlaneBuf<C>::bytes(g, k);
    if (in_step) launch_after(any::ka_plane_forward<T, TWO>, grid, threads, smem, st, g, jobs, s, f0, f1, spec, stack(g, k));
    else any::ka_plane_forward<T, TWO><<<grid, threads, smem, st>>>(g, jobs, s, f0, f1, spec, stack(g, k));
}
template <typename T, bool TWO> void plane_inverse(const AnyGrid *a, cudaStream_t st, const lfts_step_job *jobs, int nj, int s, int spec, int f0) {
    using C = typename CT<T>::type;
    const Plan &g = a->p;
    const int units = TWO ? g.n0 : ceil_div(g.n0, 2), k = stack_planes<C>(a, units, nj), ctas = ceil_div(units, k);
    launch_after(any::ka_plane_inverse<T, TWO>, dim3(ctas, nj), plane_threads(a, ctas * nj, k * g.n1 * g.n2), any::PlaneBuf<C>::bytes(g, k), st, g, jobs, s, spec, f0, stack(g, k));
}
template <typename T, int NBR> void xpass(const AnyGrid *a, cudaStream_t st, const lfts_step_job *jobs, int nj, int spec, int b0, int b1) {
    using C = typename CT<T>::type;
    const Plan &g = a->p;
    const int tj = tile_columns<C>(a, NBR, nj, a->max_smem), ctas = ceil_div(g.n1 * g.nzc, tj);
    launch_after(any::ka_xpass<T, NBR>, dim3(ctas, nj), plane_threads(a, ctas * nj, g.n0 * tj * NBR), any::TileBuf<C>::bytes(g, NBR * tj), st, g, jobs, spec, b0, b1, tj, any::div_mul(tj), any::div_mul(NBR * tj));
}
template <typename T> void steps_continuous(const AnyGrid *a, cudaStream_t st, const lfts_step_job *jobs, int nj, int s0, int nsteps) {
    using C = typename CT<T>::type;
    const Plan &g = a->p;
    const int pairs = ceil_div(g.n0, 2), km = stack_planes<C>(a, pairs, nj), mid_ctas = ceil_div(pairs, km);
    const int k = stack_planes<C>(a, g.n0, nj), ctas = ceil_div(g.n0, k);
    plane_forward<T, true>(a, st, jobs, nj, s0, FM_FAC_SQ, FM_FAC, 0);
    for (int s = s0; s < s0 + nsteps; s++) {
        xpass<T, 2>(a, st, jobs, nj, 0, 0, 1);
        launch_after(any::ka_plane_mid<T, false>, dim3(mid_ctas, nj), plane_threads(a, mid_ctas * nj, km * g.n1 * g.n2), any::PlaneBuf<C>::bytes(g, km),
                     st, g, jobs, 1, 0, stack(g, km));
        xpass<T, 1>(a, st, jobs, nj, 1, 1, 1);
        if (s + 1 < s0 + nsteps)
            launch_after(any::ka_plane_seam<T>, dim3(ctas, nj), plane_threads(a, ctas * nj, k * g.n1 * g.n2), any::PlaneBuf<C>::bytes(g, k), st,
                         g, jobs, s, stack(g, k));
        else
            plane_inverse<T, true>(a, st, jobs, nj, s, 0, 0);
    }
}
template <typename T> void steps_discrete(const AnyGrid *a, cudaStream_t st, const lfts_step_job *jobs, int nj, int s0, int nsteps, int half, int wf) {
    using C = typename CT<T>::type;
    const Plan &g = a->p;
    const int pairs = ceil_div(g.n0, 2), km = stack_planes<C>(a, pairs, nj), ctas = ceil_div(pairs, km);
    plane_forward<T, false>(a, st, jobs, nj, s0, FM_NONE, 0, 0);
    for (int s = s0; s < s0 + nsteps; s++) {
        xpass<T, 1>(a, st, jobs, nj, 0, half, half);
        if (s + 1 < s0 + nsteps)
            launch_after(any::ka_plane_mid<T, true>, dim3(ctas, nj), plane_threads(a, ctas * nj, km * g.n1 * g.n2), any::PlaneBuf<C>::bytes(g, km), st,
                         g, jobs, 0, s, stack(g, km));
        else
            plane_inverse<T, false>(a, st, jobs, nj, s, 0, wf ? FM_FAC : FM_NONE);
    }
}
template <typename T> void xforward(const AnyGrid *a, cudaStream_t st, const lfts_step_job *jobs, int nj) {
    using C = typename CT<T>::type;
    const Plan &g = a->p;
    const int tj = tile_columns<C>(a, 1, nj, a->max_smem), ctas = ceil_div(g.n1 * g.nzc, tj);
    any::ka_xpass_forward<T><<<dim3(ctas, nj), plane_threads(a, ctas * nj, g.n0 * tj), any::TileBuf<C>::bytes(g, tj), st>>>(
        g, jobs, tj, any::div_mul(tj), any::div_mul(tj));
}
template <typename T> void xstress(const AnyGrid *a, cudaStream_t st, const lfts_step_job *sj, const lfts_stress_job *jobs, int nj,
                                   const double *basis, double *partials) {
    using C = typename CT<T>::type;
    const Plan &g = a->p;
    const int tj = tile_columns<C>(a, 2, nj, a->stress_smem);
    any::ka_xstress<T><<<dim3(ceil_div(g.n1 * g.nzc, tj), nj), NTHR, any::TileBuf<C>::bytes(g, 2 * tj), st>>>(
        g, sj, jobs, basis, tj, any::div_mul(tj), any::div_mul(2 * tj), partials);
}
template <typename T> int sweep_continuous(const AnyGrid *a, cudaStream_t st, const lfts_step_job *jobs, int nj, int s0, int n, int cs) {
    const SweepShape s = sweep_shape(a, true, cs);
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at;
    cluster_config(cfg, &at, any::ka_sweep_continuous<T>, cs, nj, sweep_threads(a, s), s.smem, st);
    return (int)cudaLaunchKernelEx(&cfg, any::ka_sweep_continuous<T>, a->p, s.w, jobs, s0, n);
}
template <typename T> int sweep_discrete(const AnyGrid *a, cudaStream_t st, const lfts_step_job *jobs, int nj, int s0, int n, int half, int wf, int cs) {
    const SweepShape s = sweep_shape(a, false, cs);
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at;
    cluster_config(cfg, &at, any::ka_sweep_discrete<T>, cs, nj, sweep_threads(a, s), s.smem, st);
    return (int)cudaLaunchKernelEx(&cfg, any::ka_sweep_discrete<T>, a->p, s.w, jobs, s0, n, half, wf);
}
}  // namespace

bool any_radices(int n, std::vector<int> &r) {
    // primes above 13 go innermost (span 1: no twiddles)
    std::vector<int> big, cur;
    int m = n;
    for (int q = 17; q <= m; q += 2)
        while (m % q == 0) {
            bool prime = true;
            for (int d = 3; d * d <= q; d += 2) prime = prime && q % d;
            if (!prime) break;
            big.push_back(q);
            m /= q;
        }
    r.clear();
    if (m > 1) best_radices(m, cur, r, any::MAX_REG_RADIX);
    for (int q : big) {
        if (q > LFTS_MAX_RADIX) return false;
        r.push_back(q);
    }
    return (int)r.size() <= any::MAXF;
}

AnyGrid *any_create(int prec, const int n[3], int nsm, int max_smem, std::string &err) {
    auto *a = new AnyGrid();
    Plan &g = a->p;
    std::memset(&g, 0, sizeof g);
    // one x-plane (a 2D box): its rows become planes of one row each, so they spread over the SMs
    g.n0 = n[0] == 1 ? n[1] : n[0];
    g.n1 = n[0] == 1 ? 1 : n[1];
    g.n2 = n[2];
    g.nzc = g.n2 / 2 + 1;
    g.pitch = g.n2 | 1;
    g.M = (long long)g.n0 * g.n1 * g.n2;
    g.Mc = (long long)g.n0 * g.n1 * g.nzc;
    g.mul_n1 = any::div_mul(g.n1);
    g.mul_n2 = any::div_mul(g.n2);
    g.mul_nzc = any::div_mul(g.nzc);
    a->prec = prec;
    a->nsm = nsm;
    a->max_smem = max_smem;
    if (!(prec == 8 ? setup<double>(a, err) : setup<float>(a, err))) {
        any_destroy(a);
        return nullptr;
    }
    return a;
}
void any_destroy(AnyGrid *a) {
    if (!a) return;
    if (a->tables) cudaFree(a->tables);
    delete a;
}
void any_steps_continuous(const AnyGrid *a, cudaStream_t st, const lfts_step_job *jobs, int nj, int s0, int nsteps) {
    a->prec == 8 ? steps_continuous<double>(a, st, jobs, nj, s0, nsteps) : steps_continuous<float>(a, st, jobs, nj, s0, nsteps);
}
void any_steps_discrete(const AnyGrid *a, cudaStream_t st, const lfts_step_job *jobs, int nj, int s0, int nsteps, int half, int wf) {
    a->prec == 8 ? steps_discrete<double>(a, st, jobs, nj, s0, nsteps, half, wf) : steps_discrete<float>(a, st, jobs, nj, s0, nsteps, half, wf);
}
void any_planes_forward(const AnyGrid *a, cudaStream_t st, const lfts_step_job *jobs, int nj) {
    a->prec == 8 ? plane_forward<double, false>(a, st, jobs, nj, 0, FM_NONE, 0, 0, false) : plane_forward<float, false>(a, st, jobs, nj, 0, FM_NONE, 0, 0, false);
}
void any_xpass_forward(const AnyGrid *a, cudaStream_t st, const lfts_step_job *jobs, int nj) {
    a->prec == 8 ? xforward<double>(a, st, jobs, nj) : xforward<float>(a, st, jobs, nj);
}
int any_stress_tiles(const AnyGrid *a, int nj) {
    return ceil_div(a->p.n1 * a->p.nzc, a->prec == 8 ? tile_columns<double2>(a, 2, nj, a->stress_smem) : tile_columns<float2>(a, 2, nj, a->stress_smem));
}
void any_xstress(const AnyGrid *a, cudaStream_t st, const lfts_step_job *sj, const lfts_stress_job *jobs, int nj, const double *basis,
                 double *partials) {
    a->prec == 8 ? xstress<double>(a, st, sj, jobs, nj, basis, partials) : xstress<float>(a, st, sj, jobs, nj, basis, partials);
}
// A sweep's step costs barriers and transposes whatever the grid, then time per point
// a CTA holds; the separate passes cost four (discrete: two) launches, then time per
// point of all jobs.  Microseconds a step measured on a B200, 2 jobs, FP64 (FP32), clusters
// of 16 / separate: 84 x 48 20.6 / 26.8 (17.7 / 27.0); 256 points 16.5 / 25.0 (14.2 / 22.9);
// 24^3 25.0 / 27.8 (21.5 / 27.1); 32^3, 32 768 points, 32.4 / 30.2 (26.8 / 28.3): the lines
// cross near 1500 (2500) points a CTA.  More clusters than the device holds at once run in
// waves.  Where the rule misses the best of the sizes it is by up to a quarter, with many
// jobs on one short axis (256 points, 64 jobs: clusters of 8 19.7, of 2 16.5).
int any_sweep_size(const AnyGrid *a, bool continuous, int nj, int force) {
    const int *res = continuous ? a->clusters_cont : a->clusters_disc;
    if (force) {
        for (int k = 0; k < 5; k++)
            if (1 << k == force && res[k]) return force;
        return 0;
    }
    const bool f64 = a->prec == 8;
    const double M = (double)a->p.M, part = continuous ? 1.0 : 0.55;
    const double fixed = f64 ? 17.5 : 14.5, per_point = f64 ? 7.3e-3 : 4.8e-3;
    double best = part * (26.0 + nj * M * (f64 ? 5e-5 : 4e-5));
    int size = 0;
    for (int k = 0; k < 5; k++) {
        if (!res[k]) continue;
        const double t = part * ((nj + res[k] - 1) / res[k]) * (fixed + per_point * M / (1 << k));
        if (t < best) {
            best = t;
            size = 1 << k;
        }
    }
    return size;
}
int any_sweep_continuous(const AnyGrid *a, cudaStream_t st, const lfts_step_job *jobs, int nj, int s0, int nsteps, int cs) {
    return a->prec == 8 ? sweep_continuous<double>(a, st, jobs, nj, s0, nsteps, cs) : sweep_continuous<float>(a, st, jobs, nj, s0, nsteps, cs);
}
int any_sweep_discrete(const AnyGrid *a, cudaStream_t st, const lfts_step_job *jobs, int nj, int s0, int nsteps, int half, int wf, int cs) {
    return a->prec == 8 ? sweep_discrete<double>(a, st, jobs, nj, s0, nsteps, half, wf, cs)
                        : sweep_discrete<float>(a, st, jobs, nj, s0, nsteps, half, wf, cs);
}

}  // namespace lfts

// Pseudo-spectral step kernels for any grid extent, and the contour sweep of a
// small grid as one cluster launch (sm_100a).
//
// The passes are those of the other families (K1 plane forward, K2 x-pass, K3
// plane mid, K4 x-pass, K5 plane inverse; discrete: K1, K2, K5).  A plane here is
// ONE complex n1 x n2 transform that carries two real planes, as real and
// imaginary part: the two Richardson branches of an x-plane (K1, K5) or two
// neighbouring x-planes (K3 and the discrete step).  The half spectra of the two
// are separated, or put together, while they pass between shared memory and the
// spectrum in HBM, so rows need no pairing and odd extents no special case.
//
// ka_sweep_* run every step of a launch without leaving the SMs: a thread-block
// cluster holds one job, its CTAs a slab of x-planes and a range of (y, kz)
// columns each, and the two transposes of a step read the other CTAs' shared
// memory.  q is written once a step and nothing else reaches HBM.
#pragma once
#include "lfts_fft_any.cuh"
#include "lfts_reduce.cuh"

namespace lfts {
namespace any {

constexpr int NT_MAX = 512;

template <typename C>
struct PlaneBuf {
    C *buf, *twy, *twz;
    short *iy, *iz;  // position -> natural index
    __device__ PlaneBuf(unsigned char *raw, const Plan &g, int planes) {
        buf = (C *)raw;
        twy = buf + (size_t)planes * g.n1 * g.pitch;
        twz = twy + g.n1;
        iy = (short *)(twz + g.n2);
        iz = iy + g.n1;
        for (int i = threadIdx.x; i < g.n1; i += blockDim.x) { twy[i] = ((const C *)g.tw[1])[i]; iy[i] = g.iperm[1][i]; }
        for (int i = threadIdx.x; i < g.n2; i += blockDim.x) { twz[i] = ((const C *)g.tw[2])[i]; iz[i] = g.iperm[2][i]; }
    }
    static size_t bytes(const Plan &g, int planes) {
        return sizeof(C) * ((size_t)planes * g.n1 * g.pitch + g.n1 + g.n2) + sizeof(short) * (g.n1 + g.n2);
    }
};

// Packed planes stacked in one buffer, with the divisions of their line counts
// (prepared by the host; a CTA with fewer planes transforms the unused ones too)
struct Stack {
    int planes;
    unsigned mul_rows, mul_cols;  // division by planes * n1 and by planes * n2
};
// z lines (rows) and y lines (columns)
__device__ __forceinline__ Lines z_lines(const Plan &g, const Stack &k) {
    return {k.planes * g.n1, k.mul_rows, g.pitch, 1, 0u, 0};
}
__device__ __forceinline__ Lines y_lines(const Plan &g, const Stack &k) {
    return {k.planes * g.n2, k.mul_cols, 1, g.pitch, g.mul_n2, k.planes > 1 ? g.n1 * g.pitch - g.n2 : 0};
}
template <typename C>
__device__ __forceinline__ void plane_forward(const Plan &g, C *buf, const Stack &k, const C *twy, const C *twz) {
    transform<false>(buf, z_lines(g, k), g.ax[2], twz);
    transform<false>(buf, y_lines(g, k), g.ax[1], twy);
}
template <typename C>
__device__ __forceinline__ void plane_inverse(const Plan &g, C *buf, const Stack &k, const C *twy, const C *twz) {
    transform<true>(buf, y_lines(g, k), g.ax[1], twy);
    transform<true>(buf, z_lines(g, k), g.ax[2], twz);
}

// Half spectra of the two real planes a packed plane carries, at (ky, kz)
template <typename C>
__device__ __forceinline__ void separate(C z, C zn, C &A, C &B) {
    zn.y = -zn.y;
    split_pair(z, zn, A, B);
}
// and back: the packed values at (ky, kz) and at (-ky, -kz)
template <typename C>
__device__ __forceinline__ void join(C A, C B, C &z, C &zn) {
    z.x = A.x - B.y;
    z.y = A.y + B.x;
    zn.x = A.x + B.y;
    zn.y = B.x - A.y;
}

// real-space point of shared-memory index i over stacked planes: plane p, row y
// and column t in natural order, buffer offset o
struct Point {
    int p, y, t, o;
};
__device__ __forceinline__ Point point_at(const Plan &g, int i, const short *iy, const short *iz) {
    const int r = fdiv(i, g.mul_n2), c = i - r * g.n2;
    const int p = fdiv(r, g.mul_n1), yr = r - p * g.n1;
    return {p, iy[yr], iz[c], r * g.pitch + c};
}

// v / 3 as v times a third in two parts (a quotient of FP64 numbers costs ten times
// this).  Both parts are positive: an infinite v stays infinite.
template <typename T> __device__ __forceinline__ T third(T v) {
    constexpr T hi = sizeof(T) == 8 ? (T)0x1.5555555555555p-2 : (T)0x1.555554p-2;  // a third, rounded down
    constexpr T lo = sizeof(T) == 8 ? (T)(1.0 / 3.0 * 0x1p-54) : (T)(1.0 / 3.0 - (double)hi);
    return fma(v, hi, v * lo);
}

constexpr int U = 4;  // independent global loads a thread keeps in flight

// ------------------------------------------------------------------------
// K1.  TWO: plane x with both branches (factors fm0, fm1) -> spectra b = 0, 1.
// Otherwise planes 2p, 2p + 1 with factor fm0 -> spectrum spec_out.
template <typename T, bool TWO>
__global__ void __launch_bounds__(NT_MAX) ka_plane_forward(const __grid_constant__ Plan g, const lfts_step_job *__restrict__ jobs, int s, int fm0,
                                                           int fm1, int spec_out, Stack sk) {
    using C = typename CT<T>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PlaneBuf<C> sm(smem_raw, g, sk.planes);
    grid_wait();
    const lfts_step_job jb = jobs[blockIdx.y];
    if (jb.active && !jb.active[jb.replica]) return;
    __syncthreads();
    const int per = TWO ? 1 : 2, x0 = blockIdx.x * sk.planes * per;
    const int nx = min(sk.planes * per, g.n0 - x0), np = (nx + per - 1) / per, area = g.n1 * g.n2;
    const T *qin = (const T *)jb.in + s * jb.in_stride + (long long)x0 * area;
    const T *fac = (const T *)jb.fac + (long long)x0 * area;
    const int tot = np * area;
    for (int i0 = threadIdx.x; i0 < tot; i0 += U * blockDim.x) {
        T a[U], b[U], fa[U], fb[U];
        int o[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = i0 + u * blockDim.x;
            a[u] = b[u] = (T)0;
            fa[u] = fb[u] = (T)1;
            if (i < tot) {
                const Point pt = point_at(g, i, sm.iy, sm.iz);
                const int src = (pt.p * per * g.n1 + pt.y) * g.n2 + pt.t;
                o[u] = pt.o;
                a[u] = qin[src];
                if (fm0 != FM_NONE) fa[u] = fac[src];
                if (!TWO && pt.p * 2 + 1 < nx) {
                    b[u] = qin[src + area];
                    if (fm0 != FM_NONE) fb[u] = fac[src + area];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (i0 + u * (int)blockDim.x < tot) {
                C z;
                if (TWO) {
                    z.x = a[u] * (fm0 == FM_FAC_SQ ? fa[u] * fa[u] : fa[u]);
                    z.y = a[u] * (fm1 == FM_FAC_SQ ? fa[u] * fa[u] : fa[u]);
                } else {
                    z.x = a[u] * (fm0 == FM_FAC_SQ ? fa[u] * fa[u] : fa[u]);
                    z.y = b[u] * (fm0 == FM_FAC_SQ ? fb[u] * fb[u] : fb[u]);
                }
                sm.buf[o[u]] = z;
            }
        }
    }
    __syncthreads();
    plane_forward(g, sm.buf, sk, sm.twy, sm.twz);
    const int half = g.n1 * g.nzc;
    C *out = (C *)jb.spec + (size_t)(TWO ? 0 : spec_out) * g.Mc + (size_t)x0 * half;
    for (int i = threadIdx.x; i < np * half; i += blockDim.x) {
        const int r = fdiv(i, g.mul_nzc), kz = i - r * g.nzc;
        const int p = fdiv(r, g.mul_n1), ky = r - p * g.n1;
        const int rn = p * g.n1 + (ky ? g.n1 - ky : 0);
        C A, B;
        separate(sm.buf[r * g.pitch + kz], sm.buf[rn * g.pitch + (kz ? g.n2 - kz : 0)], A, B);
        if (TWO) {
            out[i] = A;
            out[g.Mc + i] = B;
        } else {
            const int d = (2 * p * g.n1 + ky) * g.nzc + kz;
            out[d] = A;
            if (2 * p + 1 < nx) out[d + half] = B;
        }
    }
}

// spectra -> packed planes at natural positions
template <typename C, bool TWO>
__device__ __forceinline__ void load_packed(const Plan &g, const C *__restrict__ in, C *buf, int np, int nx) {
    const int half = g.n1 * g.nzc, tot = np * half;
    for (int i0 = threadIdx.x; i0 < tot; i0 += U * blockDim.x) {
        C A[U], B[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = i0 + u * blockDim.x;
            B[u] = cmk<C>(0, 0);
            if (i < tot) {
                if (TWO) {
                    A[u] = in[i];
                    B[u] = in[g.Mc + i];
                } else {
                    const int p = fdiv(fdiv(i, g.mul_nzc), g.mul_n1);
                    A[u] = in[i + p * half];
                    if (2 * p + 1 < nx) B[u] = in[i + (p + 1) * half];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = i0 + u * blockDim.x;
            if (i < tot) {
                const int r = fdiv(i, g.mul_nzc), kz = i - r * g.nzc;
                const int p = fdiv(r, g.mul_n1), ky = r - p * g.n1;
                C z, zn;
                join(A[u], B[u], z, zn);
                buf[r * g.pitch + kz] = z;
                if (kz && 2 * kz != g.n2) buf[(p * g.n1 + (ky ? g.n1 - ky : 0)) * g.pitch + g.n2 - kz] = zn;
            }
        }
    }
}

// ------------------------------------------------------------------------
// K3: inverse zy of planes 2p, 2p + 1, multiply by fac^2, forward zy, in place
// (SEAM: the discrete step's seam, K5 of step s and K1 of step s + 1: the factor is fac
// and the product, q', also goes to memory)
template <typename T, bool SEAM>
__global__ void __launch_bounds__(NT_MAX) ka_plane_mid(const __grid_constant__ Plan g, const lfts_step_job *__restrict__ jobs, int spec_idx, int s,
                                                       Stack sk) {
    using C = typename CT<T>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PlaneBuf<C> sm(smem_raw, g, sk.planes);
    const lfts_step_job jb = jobs[blockIdx.y];
    grid_wait();
    if (jb.active && !jb.active[jb.replica]) return;
    const int x0 = blockIdx.x * sk.planes * 2, nx = min(sk.planes * 2, g.n0 - x0), np = (nx + 1) / 2;
    const int area = g.n1 * g.n2, half = g.n1 * g.nzc;
    C *spec = (C *)jb.spec + (size_t)spec_idx * g.Mc + (size_t)x0 * half;
    load_packed<C, false>(g, spec, sm.buf, np, nx);
    __syncthreads();
    plane_inverse(g, sm.buf, sk, sm.twy, sm.twz);
    const T *fac = (const T *)jb.fac + (long long)x0 * area;
    T *qout = SEAM ? (T *)jb.out + s * jb.out_stride + (long long)x0 * area : nullptr;
    for (int i = threadIdx.x; i < np * area; i += blockDim.x) {
        const Point pt = point_at(g, i, sm.iy, sm.iz);
        const int src = (2 * pt.p * g.n1 + pt.y) * g.n2 + pt.t;
        const T ea = fac[src], eb = 2 * pt.p + 1 < nx ? fac[src + area] : (T)0;
        C z = sm.buf[pt.o];
        z.x *= SEAM ? ea : ea * ea;
        z.y *= SEAM ? eb : eb * eb;
        if (SEAM) {
            qout[src] = z.x;
            if (2 * pt.p + 1 < nx) qout[src + area] = z.y;
        }
        sm.buf[pt.o] = z;
    }
    __syncthreads();
    plane_forward(g, sm.buf, sk, sm.twy, sm.twz);
    for (int i = threadIdx.x; i < np * half; i += blockDim.x) {
        const int r = fdiv(i, g.mul_nzc), kz = i - r * g.nzc;
        const int p = fdiv(r, g.mul_n1), ky = r - p * g.n1;
        C A, B;
        separate(sm.buf[r * g.pitch + kz], sm.buf[(p * g.n1 + (ky ? g.n1 - ky : 0)) * g.pitch + (kz ? g.n2 - kz : 0)], A, B);
        const int d = (2 * p * g.n1 + ky) * g.nzc + kz;
        spec[d] = A;
        if (2 * p + 1 < nx) spec[d + half] = B;
    }
}

// ------------------------------------------------------------------------
// K5.  TWO: q' = (4 e_h v_half - e_h^2 v_full) / 3 of plane x.  Otherwise
// q' = v * factor(fm0) of planes 2p, 2p + 1.
template <typename T, bool TWO>
__global__ void __launch_bounds__(NT_MAX) ka_plane_inverse(const __grid_constant__ Plan g, const lfts_step_job *__restrict__ jobs, int s, int spec_in,
                                                           int fm0, Stack sk) {
    using C = typename CT<T>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PlaneBuf<C> sm(smem_raw, g, sk.planes);
    const lfts_step_job jb = jobs[blockIdx.y];
    grid_wait();
    if (jb.active && !jb.active[jb.replica]) return;
    const int per = TWO ? 1 : 2, x0 = blockIdx.x * sk.planes * per;
    const int nx = min(sk.planes * per, g.n0 - x0), np = (nx + per - 1) / per, area = g.n1 * g.n2, half = g.n1 * g.nzc;
    load_packed<C, TWO>(g, (const C *)jb.spec + (size_t)(TWO ? 0 : spec_in) * g.Mc + (size_t)x0 * half, sm.buf, np, nx);
    __syncthreads();
    plane_inverse(g, sm.buf, sk, sm.twy, sm.twz);
    const T *fac = (const T *)jb.fac + (long long)x0 * area;
    T *qout = (T *)jb.out + s * jb.out_stride + (long long)x0 * area;
    for (int i = threadIdx.x; i < np * area; i += blockDim.x) {
        const Point pt = point_at(g, i, sm.iy, sm.iz);
        const int src = (pt.p * per * g.n1 + pt.y) * g.n2 + pt.t;
        const C z = sm.buf[pt.o];
        if (TWO) {
            const T eh = fac[src];
            qout[src] = third((T)4 * eh * z.y - eh * eh * z.x);
        } else {
            qout[src] = z.x * fac_value(fm0, fac, src);
            if (2 * pt.p + 1 < nx) qout[src + area] = z.y * fac_value(fm0, fac, src + area);
        }
    }
}

// ------------------------------------------------------------------------
// The seam between two steps of a sweep: K5 of step s and K1 of step s + 1
template <typename T>
__global__ void __launch_bounds__(NT_MAX) ka_plane_seam(const __grid_constant__ Plan g, const lfts_step_job *__restrict__ jobs, int s,
                                                        Stack sk) {
    using C = typename CT<T>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PlaneBuf<C> sm(smem_raw, g, sk.planes);
    const lfts_step_job jb = jobs[blockIdx.y];
    grid_wait();
    if (jb.active && !jb.active[jb.replica]) return;
    const int x0 = blockIdx.x * sk.planes, np = min(sk.planes, g.n0 - x0), area = g.n1 * g.n2, half = g.n1 * g.nzc;
    C *spec = (C *)jb.spec + (size_t)x0 * half;
    load_packed<C, true>(g, spec, sm.buf, np, np);
    __syncthreads();
    plane_inverse(g, sm.buf, sk, sm.twy, sm.twz);
    const T *fac = (const T *)jb.fac + (long long)x0 * area;
    T *qout = (T *)jb.out + s * jb.out_stride + (long long)x0 * area;
    for (int i = threadIdx.x; i < np * area; i += blockDim.x) {
        const Point pt = point_at(g, i, sm.iy, sm.iz);
        const int src = (pt.p * g.n1 + pt.y) * g.n2 + pt.t;
        const T eh = fac[src];
        C z = sm.buf[pt.o];
        const T q = third((T)4 * eh * z.y - eh * eh * z.x);
        qout[src] = q;
        z.x = q * (eh * eh);
        z.y = q * eh;
        sm.buf[pt.o] = z;
    }
    __syncthreads();
    plane_forward(g, sm.buf, sk, sm.twy, sm.twz);
    for (int i = threadIdx.x; i < np * half; i += blockDim.x) {
        const int r = fdiv(i, g.mul_nzc), kz = i - r * g.nzc;
        const int p = fdiv(r, g.mul_n1), ky = r - p * g.n1;
        C A, B;
        separate(sm.buf[r * g.pitch + kz], sm.buf[(p * g.n1 + (ky ? g.n1 - ky : 0)) * g.pitch + (kz ? g.n2 - kz : 0)], A, B);
        spec[i] = A;
        spec[g.Mc + i] = B;
    }
}

// ------------------------------------------------------------------------
// Tiles of TJ (y, kz) columns, NBR spectra side by side: rows x, NBR * TJ wide
template <typename C>
struct TileBuf {
    C *tile, *twx;
    short *px;  // natural index -> position
    __device__ TileBuf(unsigned char *raw, const Plan &g, int width) {
        tile = (C *)raw;
        twx = tile + (size_t)g.n0 * width;
        px = (short *)(twx + g.n0);
        for (int i = threadIdx.x; i < g.n0; i += blockDim.x) { twx[i] = ((const C *)g.tw[0])[i]; px[i] = g.perm[0][i]; }
    }
    static size_t bytes(const Plan &g, int width) {
        return sizeof(C) * ((size_t)g.n0 * width + g.n0) + sizeof(short) * g.n0;
    }
};
template <typename C, int NBR>
__device__ __forceinline__ void load_tile(const Plan &g, const C *__restrict__ spec, TileBuf<C> &sm, int j0, int nj, int TJ, unsigned mul_tj) {
    const long long plane = (long long)g.n1 * g.nzc;
    const int tot = g.n0 * TJ;
    for (int i0 = threadIdx.x; i0 < tot; i0 += U * blockDim.x) {
        C a[U], b[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = i0 + u * blockDim.x;
            a[u] = b[u] = cmk<C>(0, 0);
            if (i < tot) {
                const int x = fdiv(i, mul_tj), jj = i - x * TJ;
                if (jj < nj) {
                    a[u] = spec[x * plane + j0 + jj];
                    if (NBR == 2) b[u] = spec[g.Mc + x * plane + j0 + jj];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = i0 + u * blockDim.x;
            if (i < tot) {
                const int x = fdiv(i, mul_tj), jj = i - x * TJ;
                C *d = sm.tile + sm.px[x] * (NBR * TJ) + jj;
                d[0] = a[u];
                if (NBR == 2) d[TJ] = b[u];
            }
        }
    }
}

// K2 / K4: x-transform, bond tables, inverse
template <typename T, int NBR>
__global__ void __launch_bounds__(NT_MAX) ka_xpass(const __grid_constant__ Plan g, const lfts_step_job *__restrict__ jobs, int spec_in, int bsel0,
                                                   int bsel1, int TJ, unsigned mul_tj, unsigned mul_w) {
    using C = typename CT<T>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TileBuf<C> sm(smem_raw, g, NBR * TJ);
    const lfts_step_job jb = jobs[blockIdx.y];
    grid_wait();
    if (jb.active && !jb.active[jb.replica]) return;
    __syncthreads();
    const int plane = g.n1 * g.nzc, j0 = blockIdx.x * TJ, nj = min(TJ, plane - j0);
    C *spec = (C *)jb.spec + (size_t)spec_in * g.Mc;
    load_tile<C, NBR>(g, spec, sm, j0, nj, TJ, mul_tj);
    __syncthreads();
    const Lines lx = {NBR * TJ, mul_w, 1, NBR * TJ, 0u, 0};
    transform<false>(sm.tile, lx, g.ax[0], sm.twx);
    const T *bt0 = (const T *)(bsel0 ? jb.bond_half : jb.bond), *bt1 = (const T *)(bsel1 ? jb.bond_half : jb.bond);
    for (int i = threadIdx.x; i < g.n0 * TJ; i += blockDim.x) {
        const int x = fdiv(i, mul_tj), jj = i - x * TJ;
        if (jj < nj) {
            const long long k = (long long)x * plane + j0 + jj;
            C *d = sm.tile + x * (NBR * TJ) + jj;
            const T b0 = bt0[k];
            d[0].x *= b0;
            d[0].y *= b0;
            if (NBR == 2) {
                const T b1 = bt1[k];
                d[TJ].x *= b1;
                d[TJ].y *= b1;
            }
        }
    }
    __syncthreads();
    transform<true>(sm.tile, lx, g.ax[0], sm.twx);
    for (int i = threadIdx.x; i < g.n0 * TJ; i += blockDim.x) {
        const int x = fdiv(i, mul_tj), jj = i - x * TJ;
        if (jj < nj) {
            const C *d = sm.tile + sm.px[x] * (NBR * TJ) + jj;
            spec[(long long)x * plane + j0 + jj] = d[0];
            if (NBR == 2) spec[g.Mc + (long long)x * plane + j0 + jj] = d[TJ];
        }
    }
}

// Forward x-transform only: completes a 3D real transform
template <typename T>
__global__ void __launch_bounds__(NT_MAX) ka_xpass_forward(const __grid_constant__ Plan g, const lfts_step_job *__restrict__ jobs, int TJ, unsigned mul_tj, unsigned mul_w) {
    using C = typename CT<T>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TileBuf<C> sm(smem_raw, g, TJ);
    const lfts_step_job jb = jobs[blockIdx.y];
    if (jb.active && !jb.active[jb.replica]) return;
    __syncthreads();
    const int plane = g.n1 * g.nzc, j0 = blockIdx.x * TJ, nj = min(TJ, plane - j0);
    C *spec = (C *)jb.spec;
    load_tile<C, 1>(g, spec, sm, j0, nj, TJ, mul_tj);
    __syncthreads();
    const Lines lx = {TJ, mul_w, 1, TJ, 0u, 0};
    transform<false>(sm.tile, lx, g.ax[0], sm.twx);
    for (int i = threadIdx.x; i < g.n0 * TJ; i += blockDim.x) {
        const int x = fdiv(i, mul_tj), jj = i - x * TJ;
        if (jj < nj) spec[(long long)x * plane + j0 + jj] = sm.tile[x * TJ + jj];
    }
}

// Stress of one (q1, q2) pair per job: x-transform of both zy spectra, then
// sum_k Re(q1 q2*) basis_d(k).  Blocks of NTHR threads (the reductions' size).
template <typename T>
__global__ void __launch_bounds__(NTHR) ka_xstress(const __grid_constant__ Plan g, const lfts_step_job *__restrict__ sj,
                                                   const lfts_stress_job *__restrict__ jobs, const double *__restrict__ basis,
                                                   int TJ, unsigned mul_tj, unsigned mul_w, double *partials) {
    using C = typename CT<T>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double sh[2 * NWARP];
    TileBuf<C> sm(smem_raw, g, 2 * TJ);
    const int job = blockIdx.y;
    const C *spec = (const C *)sj[2 * job].spec;  // two consecutive Mc slots
    const T *bond = (const T *)jobs[job].bond;
    __syncthreads();
    const int plane = g.n1 * g.nzc, j0 = blockIdx.x * TJ, nj = min(TJ, plane - j0);
    load_tile<C, 2>(g, spec, sm, j0, nj, TJ, mul_tj);
    __syncthreads();
    const Lines lx = {2 * TJ, mul_w, 1, 2 * TJ, 0u, 0};
    transform<false>(sm.tile, lx, g.ax[0], sm.twx);
    Acc<T> acc[3];
    for (int i = threadIdx.x; i < g.n0 * TJ; i += blockDim.x) {
        const int x = fdiv(i, mul_tj), jj = i - x * TJ;
        if (jj < nj) {
            const long long k = (long long)x * plane + j0 + jj;
            const C A = sm.tile[x * (2 * TJ) + jj], B = sm.tile[x * (2 * TJ) + TJ + jj];
            double co = (double)A.x * (double)B.x + (double)A.y * (double)B.y;
            if (bond) co *= (double)bond[k] * (double)g.M;  // tables carry 1/M
            acc[0].add(co * basis[k]);
            acc[1].add(co * basis[g.Mc + k]);
            acc[2].add(co * basis[2 * g.Mc + k]);
        }
    }
    for (int d = 0; d < 3; d++) {
        const double v = acc[d].block(sh);
        if (threadIdx.x == 0) partials[((long long)job * gridDim.x + blockIdx.x) * 3 + d] = v;
    }
}

// ------------------------------------------------------------------------
// Cluster sweeps.  rank r of the cluster holds x-planes [r XB, r XB + XB) and
// columns [r JB, r JB + JB).
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// all threads of all CTAs of the cluster; orders their shared-memory accesses
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ unsigned remote(const void *p, int rank) {
    unsigned a = (unsigned)__cvta_generic_to_shared(p), r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ double2 ld_remote(unsigned a, double2) {
    double2 v;
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ float2 ld_remote(unsigned a, float2) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
    return v;
}

template <typename C>
struct SweepBuf {
    C *pl, *col, *twx, *twy, *twz;
    short *px, *iy, *iz;
    // planes: packed planes of the slab; width: columns side by side in col
    __device__ SweepBuf(unsigned char *raw, const Plan &g, int planes, int width) {
        pl = (C *)raw;
        col = pl + (size_t)planes * g.n1 * g.pitch;
        twx = col + (size_t)g.n0 * width;
        twy = twx + g.n0;
        twz = twy + g.n1;
        px = (short *)(twz + g.n2);
        iy = px + g.n0;
        iz = iy + g.n1;
        for (int i = threadIdx.x; i < g.n0; i += blockDim.x) { twx[i] = ((const C *)g.tw[0])[i]; px[i] = g.perm[0][i]; }
        for (int i = threadIdx.x; i < g.n1; i += blockDim.x) { twy[i] = ((const C *)g.tw[1])[i]; iy[i] = g.iperm[1][i]; }
        for (int i = threadIdx.x; i < g.n2; i += blockDim.x) { twz[i] = ((const C *)g.tw[2])[i]; iz[i] = g.iperm[2][i]; }
    }
    static size_t bytes(const Plan &g, int planes, int width) {
        return sizeof(C) * ((size_t)planes * g.n1 * g.pitch + (size_t)g.n0 * width + g.n0 + g.n1 + g.n2) +
               sizeof(short) * (g.n0 + g.n1 + g.n2);
    }
};

// The shape of a sweep, its divisions prepared by the host
struct Sweep {
    int XB, JB, width;   // planes and columns a CTA, columns side by side in col
    unsigned mul_xb, mul_jb, mul_width;
    Stack all, half;     // every plane packed by itself; planes packed in pairs
};

// slab -> columns.  PER = 1: every plane is packed by itself and gives the columns of
// both branches (b at jj, b' at JB + jj); PER = 2: planes 2p, 2p + 1 packed, one branch
// at column offset coff.
template <typename C, int PER>
__device__ __forceinline__ void pull_columns(const Plan &g, const SweepBuf<C> &sm, const Sweep &w, int j0, int nj, int coff) {
    const int tot = g.n0 * w.JB;
    const C zero = cmk<C>(0, 0);
    for (int i0 = threadIdx.x; i0 < tot; i0 += U * blockDim.x) {
        C z[U], zn[U];
        int d[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = i0 + u * blockDim.x;
            const int x = fdiv(i, w.mul_jb), jj = i - x * w.JB;
            d[u] = -1;
            if (i < tot && jj < nj) {
                const int j = j0 + jj, ky = fdiv(j, g.mul_nzc), kz = j - ky * g.nzc;
                const int r = fdiv(x, w.mul_xb), xl = x - r * w.XB;
                const int row = (PER == 1 ? xl : xl >> 1) * g.n1;
                z[u] = ld_remote(remote(sm.pl + (row + ky) * g.pitch + kz, r), zero);
                zn[u] = ld_remote(remote(sm.pl + (row + (ky ? g.n1 - ky : 0)) * g.pitch + (kz ? g.n2 - kz : 0), r), zero);
                d[u] = (sm.px[x] * w.width + jj) * 2 + (PER == 1 ? 0 : xl & 1);
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (d[u] >= 0) {
                C A, B;
                separate(z[u], zn[u], A, B);
                C *o = sm.col + (d[u] >> 1);
                if (PER == 1) {
                    o[0] = A;
                    o[w.JB] = B;
                } else {
                    o[coff] = d[u] & 1 ? B : A;
                }
            }
        }
    }
}
// columns -> packed planes of the slab (nx planes from x0), natural positions
template <typename C, int PER>
__device__ __forceinline__ void pull_planes(const Plan &g, const SweepBuf<C> &sm, const Sweep &w, int x0, int nx, int coff) {
    const int half = g.n1 * g.nzc, tot = (nx + PER - 1) / PER * half;
    const C zero = cmk<C>(0, 0);
    for (int i0 = threadIdx.x; i0 < tot; i0 += U * blockDim.x) {
        C A[U], B[U];
        int d[U], dn[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = i0 + u * blockDim.x;
            A[u] = B[u] = zero;
            d[u] = dn[u] = -1;
            if (i < tot) {
                const int rw = fdiv(i, g.mul_nzc), kz = i - rw * g.nzc;
                const int p = fdiv(rw, g.mul_n1), ky = rw - p * g.n1, j = i - p * half;
                const int r = fdiv(j, w.mul_jb), jj = j - r * w.JB;
                const int x = x0 + p * PER;
                const auto a = remote(sm.col + sm.px[x] * w.width + coff + jj, r);
                A[u] = ld_remote(a, zero);
                if (PER == 1) B[u] = ld_remote(a + w.JB * (unsigned)sizeof(C), zero);
                else if (p * 2 + 1 < nx) B[u] = ld_remote(remote(sm.col + sm.px[x + 1] * w.width + coff + jj, r), zero);
                d[u] = rw * g.pitch + kz;
                if (kz && 2 * kz != g.n2) dn[u] = (p * g.n1 + (ky ? g.n1 - ky : 0)) * g.pitch + g.n2 - kz;
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (d[u] >= 0) {
                C z, zn;
                join(A[u], B[u], z, zn);
                sm.pl[d[u]] = z;
                if (dn[u] >= 0) sm.pl[dn[u]] = zn;
            }
        }
    }
}
// x-transform of the columns from coff, bond tables, inverse.  TWO: the columns of
// both branches with their own tables.
template <typename C, typename T, bool TWO>
__device__ __forceinline__ void columns(const Plan &g, const SweepBuf<C> &sm, const Sweep &w, int j0, int nj, int coff,
                                        const T *__restrict__ bond, const T *__restrict__ bond2) {
    const Lines ln = {TWO ? w.width : w.JB, TWO ? w.mul_width : w.mul_jb, 1, w.width, 0u, 0};
    transform<false>(sm.col + coff, ln, g.ax[0], sm.twx);
    const int plane = g.n1 * g.nzc;
    for (int i = threadIdx.x; i < g.n0 * w.JB; i += blockDim.x) {
        const int x = fdiv(i, w.mul_jb), jj = i - x * w.JB;
        if (jj < nj) {
            const int k = x * plane + j0 + jj;
            C *d = sm.col + x * w.width + coff + jj;
            const T b = bond[k];
            d->x *= b;
            d->y *= b;
            if (TWO) {
                const T b2 = bond2[k];
                d[w.JB].x *= b2;
                d[w.JB].y *= b2;
            }
        }
    }
    __syncthreads();
    transform<true>(sm.col + coff, ln, g.ax[0], sm.twx);
}

// Continuous (Richardson) chains: steps s0 .. s0 + nsteps - 1 of every job.  Step
// s + 1 starts from what step s wrote (out of s is in of s + 1).
template <typename T>
__global__ void __launch_bounds__(NT_MAX, 1) ka_sweep_continuous(const __grid_constant__ Plan g, const __grid_constant__ Sweep w,
                                                                 const lfts_step_job *__restrict__ jobs, int s0, int nsteps) {
    using C = typename CT<T>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SweepBuf<C> sm(smem_raw, g, w.XB, w.width);
    const lfts_step_job jb = jobs[blockIdx.y];
    if (jb.active && !jb.active[jb.replica]) return;  // the whole cluster: its CTAs share the job
    __syncthreads();
    const int rank = (int)cluster_rank(), area = g.n1 * g.n2;
    const int x0 = rank * w.XB, nx = max(0, min(w.XB, g.n0 - x0)), np2 = (nx + 1) / 2;
    const int j0 = rank * w.JB, nj = max(0, min(w.JB, g.n1 * g.nzc - j0));
    const T *fac = (const T *)jb.fac + (long long)x0 * area;
    const T *bond = (const T *)jb.bond, *bond_half = (const T *)jb.bond_half;
    const T *qin = (const T *)jb.in + s0 * jb.in_stride + (long long)x0 * area;
    for (int i = threadIdx.x; i < nx * area; i += blockDim.x) {
        const Point pt = point_at(g, i, sm.iy, sm.iz);
        const int src = (pt.p * g.n1 + pt.y) * g.n2 + pt.t;
        const T q = qin[src], e = fac[src];
        C z;
        z.x = q * (e * e);
        z.y = q * e;
        sm.pl[pt.o] = z;
    }
    __syncthreads();
    for (int s = s0; s < s0 + nsteps; s++) {
        plane_forward(g, sm.pl, w.all, sm.twy, sm.twz);
        cluster_sync();
        pull_columns<C, 1>(g, sm, w, j0, nj, 0);
        __syncthreads();
        columns<C, T, true>(g, sm, w, j0, nj, 0, bond, bond_half);
        cluster_sync();
        pull_planes<C, 2>(g, sm, w, x0, nx, w.JB);  // the half-step branch only
        __syncthreads();
        plane_inverse(g, sm.pl, w.half, sm.twy, sm.twz);
        for (int i = threadIdx.x; i < np2 * area; i += blockDim.x) {
            const Point pt = point_at(g, i, sm.iy, sm.iz);
            const int src = (2 * pt.p * g.n1 + pt.y) * g.n2 + pt.t;
            const T ea = fac[src], eb = 2 * pt.p + 1 < nx ? fac[src + area] : (T)0;
            C z = sm.pl[pt.o];
            z.x *= ea * ea;
            z.y *= eb * eb;
            sm.pl[pt.o] = z;
        }
        __syncthreads();
        plane_forward(g, sm.pl, w.half, sm.twy, sm.twz);
        cluster_sync();
        pull_columns<C, 2>(g, sm, w, j0, nj, w.JB);
        __syncthreads();
        columns<C, T, false>(g, sm, w, j0, nj, w.JB, bond_half, bond_half);
        cluster_sync();
        pull_planes<C, 1>(g, sm, w, x0, nx, 0);
        __syncthreads();
        plane_inverse(g, sm.pl, w.all, sm.twy, sm.twz);
        T *qout = (T *)jb.out + s * jb.out_stride + (long long)x0 * area;
        for (int i = threadIdx.x; i < nx * area; i += blockDim.x) {
            const Point pt = point_at(g, i, sm.iy, sm.iz);
            const int src = (pt.p * g.n1 + pt.y) * g.n2 + pt.t;
            const T eh = fac[src];
            C z = sm.pl[pt.o];
            const T q = third((T)4 * eh * z.y - eh * eh * z.x);
            qout[src] = q;
            z.x = q * (eh * eh);
            z.y = q * eh;
            sm.pl[pt.o] = z;
        }
        __syncthreads();
    }
    cluster_sync();  // no CTA leaves while another still reads its columns
}

// Discrete chains (and half-bond steps): q' = factor * conv(q, bond)
template <typename T>
__global__ void __launch_bounds__(NT_MAX, 1) ka_sweep_discrete(const __grid_constant__ Plan g, const __grid_constant__ Sweep w,
                                                               const lfts_step_job *__restrict__ jobs, int s0, int nsteps,
                                                               int half_bond, int with_fac) {
    using C = typename CT<T>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SweepBuf<C> sm(smem_raw, g, w.half.planes, w.JB);
    const lfts_step_job jb = jobs[blockIdx.y];
    if (jb.active && !jb.active[jb.replica]) return;
    __syncthreads();
    const int rank = (int)cluster_rank(), area = g.n1 * g.n2;
    const int x0 = rank * w.XB, nx = max(0, min(w.XB, g.n0 - x0)), np2 = (nx + 1) / 2;
    const int j0 = rank * w.JB, nj = max(0, min(w.JB, g.n1 * g.nzc - j0));
    const T *fac = (const T *)jb.fac + (long long)x0 * area;
    const T *bond = (const T *)(half_bond ? jb.bond_half : jb.bond);
    const T *qin = (const T *)jb.in + s0 * jb.in_stride + (long long)x0 * area;
    for (int i = threadIdx.x; i < np2 * area; i += blockDim.x) {
        const Point pt = point_at(g, i, sm.iy, sm.iz);
        const int src = (2 * pt.p * g.n1 + pt.y) * g.n2 + pt.t;
        C z;
        z.x = qin[src];
        z.y = 2 * pt.p + 1 < nx ? qin[src + area] : (T)0;
        sm.pl[pt.o] = z;
    }
    __syncthreads();
    for (int s = s0; s < s0 + nsteps; s++) {
        plane_forward(g, sm.pl, w.half, sm.twy, sm.twz);
        cluster_sync();
        pull_columns<C, 2>(g, sm, w, j0, nj, 0);
        __syncthreads();
        columns<C, T, false>(g, sm, w, j0, nj, 0, bond, bond);
        cluster_sync();
        pull_planes<C, 2>(g, sm, w, x0, nx, 0);
        __syncthreads();
        plane_inverse(g, sm.pl, w.half, sm.twy, sm.twz);
        T *qout = (T *)jb.out + s * jb.out_stride + (long long)x0 * area;
        for (int i = threadIdx.x; i < np2 * area; i += blockDim.x) {
            const Point pt = point_at(g, i, sm.iy, sm.iz);
            const int src = (2 * pt.p * g.n1 + pt.y) * g.n2 + pt.t;
            C z = sm.pl[pt.o];
            if (with_fac) z.x *= fac[src];
            qout[src] = z.x;
            if (2 * pt.p + 1 < nx) {
                if (with_fac) z.y *= fac[src + area];
                qout[src + area] = z.y;
            }
            sm.pl[pt.o] = z;
        }
        __syncthreads();
    }
    cluster_sync();
}

}  // namespace any
}  // namespace lfts

// Shared-memory line transforms for any grid extent (sm_100a).
//
// A line of n = r0 r1 ... elements is transformed in place, one radix a stage:
//   forward (DIT): input at digit-reversed positions -> natural-order output,
//   inverse (DIF): natural-order input -> output at digit-reversed positions,
// so real space sits at permuted positions, spectra at natural ones, and no
// pass over memory only permutes.  A thread holds one butterfly: R complex
// values in registers, R shared-memory loads and stores a stage.
//
// What bounds these transforms on the grids that use them is the number of
// stages (each a shared-memory round trip and a barrier) and, with extents
// known only at run time, the index arithmetic.  Hence
//   * radices up to 13 and 16 in registers: of the 112 extents from 2 to 256 with
//     factors up to 13, 78 take one or two stages and 34 (75, 98, 105, 125 ...) three;
//   * divisions by run-time extents as one multiply-high with a factor the
//     host prepared, and twiddle indices that need no remainder;
//   * lines vary fastest over threads, with an odd pitch between rows, so the
//     accesses of a warp fall on different banks along rows and columns;
//   * a prime factor above 13 as cosine and sine sums of the pairs (j, R - j),
//     one pair of outputs a thread (a quarter of the direct sum's operations).
#pragma once
#include "lfts_fft.cuh"

namespace lfts {
namespace any {

constexpr int MAXF = 10;
constexpr int MAX_REG_RADIX = 16;

// t / d for 0 <= t, t * d < 2^32: mul = floor(2^32 / d) + 1, or 0 for d = 1
__host__ __device__ __forceinline__ unsigned div_mul(unsigned d) { return d <= 1 ? 0u : (unsigned)(0x100000000ull / d + 1); }
__device__ __forceinline__ int fdiv(int t, unsigned mul) { return mul ? (int)__umulhi((unsigned)t, mul) : t; }

// One axis, outermost radix first: n = radix[0] * ... * radix[nf-1].  Everything a
// stage needs that the host can divide is divided there.
struct Stage {
    int radix, span;    // span: product of the radices inside this one
    unsigned span_mul;  // division by the span
    int nbf, twstep;    // butterflies a line, n / (span * radix)
};
struct Axis {
    int n, nf;
    Stage st[MAXF];
};

// The grid as the kernels see it: x-planes of n1 x n2 points (n2 fastest).  A
// 2D box is n0 planes of one row, so that its rows spread over the SMs.
struct Plan {
    int n0, n1, n2, nzc, pitch;  // pitch: n2 made odd, complex elements between rows in shared memory
    long long M, Mc;
    Axis ax[3];
    const void *tw[3];       // exp(-2 pi i j / n), n entries, precision T
    const short *perm[3];    // natural index -> position
    const short *iperm[3];   // position -> natural index
    unsigned mul_n1, mul_n2, mul_nzc;
};

// A set of lines in shared memory: line l starts at l * ls + (l / inner) * extra
struct Lines {
    int nl;
    unsigned nl_mul;
    int ls, es;
    unsigned inner_mul;
    int extra;
    __device__ __forceinline__ int off(int l) const { return l * ls + (extra ? fdiv(l, inner_mul) * extra : 0); }
};

// cos(2 pi k / R) and sin(2 pi k / R) of the odd and composite register radices
__host__ __device__ constexpr double cos_r(int R, int k) {
    k %= R;
    if (2 * k > R) k = R - k;
    if (k == 0) return 1.0;
    if (R == 7) return k == 1 ? 0.62348980185873353052500488400424 : k == 2 ? -0.22252093395631440428890256449679 : -0.90096886790241912623610231950745;
    if (R == 9) return k == 1 ? 0.76604444311897803520239265055542 : k == 2 ? 0.17364817766693034885171662676931 : k == 3 ? -0.5 : -0.93969262078590838405410927732473;
    if (R == 11) return k == 1 ? 0.84125353283118116886181164891937 : k == 2 ? 0.41541501300188642552927414922962 : k == 3 ? -0.14231483827328514044379266861637
                      : k == 4 ? -0.65486073394528506405692507246629 : -0.95949297361449738989036805706633;
    if (R == 13) return k == 1 ? 0.88545602565320989590037552201510 : k == 2 ? 0.56806474673115580251180755912752 : k == 3 ? 0.12053668025532305334906768745254
                      : k == 4 ? -0.35460488704253562596963789260002 : k == 5 ? -0.74851074817110109863463059970135 : -0.97094181742605202715698227629379;
    return k == 1 ? 0.92387953251128675612818318939679 : k == 2 ? 0.70710678118654752440084436210485 : k == 3 ? 0.38268343236508977172845998403040
         : k == 4 ? 0.0 : k == 5 ? -0.38268343236508977172845998403040 : k == 6 ? -0.70710678118654752440084436210485
         : k == 7 ? -0.92387953251128675612818318939679 : -1.0;  // R == 16
}
__host__ __device__ constexpr double sin_r(int R, int k) {
    k %= R;
    double s = 1.0;
    if (2 * k > R) { k = R - k; s = -1.0; }
    if (k == 0) return 0.0;
    if (R == 7) return s * (k == 1 ? 0.78183148246802980870844452667406 : k == 2 ? 0.97492791218182360701813168299393 : 0.43388373911755812047576833284836);
    if (R == 9) return s * (k == 1 ? 0.64278760968653932632264340990726 : k == 2 ? 0.98480775301220805936674302458952 : k == 3 ? 0.86602540378443864676372317075294 : 0.34202014332566873304409961468226);
    if (R == 11) return s * (k == 1 ? 0.54064081745559758210763595431869 : k == 2 ? 0.90963199535451837141171538307903 : k == 3 ? 0.98982144188093273237609203777672
                           : k == 4 ? 0.75574957435425828377403584397234 : 0.28173255684142969771141791534662);
    if (R == 13) return s * (k == 1 ? 0.46472317204376854565601533513310 : k == 2 ? 0.82298386589365639457961742343938 : k == 3 ? 0.99270887409805399280075164949252
                           : k == 4 ? 0.93501624268541482343978459983783 : k == 5 ? 0.66312265824079520237678549266677 : 0.23931566428755776714875372626021);
    return s * (k == 1 ? 0.38268343236508977172845998403040 : k == 2 ? 0.70710678118654752440084436210485 : k == 3 ? 0.92387953251128675612818318939679
              : k == 4 ? 1.0 : k == 5 ? 0.92387953251128675612818318939679 : k == 6 ? 0.70710678118654752440084436210485
              : k == 7 ? 0.38268343236508977172845998403040 : 0.0);  // R == 16
}
__host__ __device__ constexpr int inv_mod(int a, int m) {
    for (int x = 1; x < m; x++)
        if ((a * x) % m == 1) return x;
    return 1;
}

// ---- forward DFT of R registers, natural order in and out
template <int R, typename C> __device__ __forceinline__ void dft(C *a);

// odd prime: sums and differences of the pairs (j, R - j)
template <int R, typename C> __device__ __forceinline__ void dft_odd(C *a) {
    using T = decltype(a[0].x);
    constexpr int H = (R - 1) / 2;
    C s[H], d[H];
#pragma unroll
    for (int j = 0; j < H; j++) {
        s[j] = cadd(a[j + 1], a[R - 1 - j]);
        d[j] = csub(a[j + 1], a[R - 1 - j]);
    }
    const C a0 = a[0];
#pragma unroll
    for (int j = 0; j < H; j++) a[0] = cadd(a[0], s[j]);
#pragma unroll
    for (int k = 1; k <= H; k++) {
        C m = a0, n = cmk<C>(0, 0);
#pragma unroll
        for (int j = 1; j <= H; j++) {
            const T c = (T)cos_r(R, (j * k) % R), w = (T)sin_r(R, (j * k) % R);
            m.x += c * s[j - 1].x;
            m.y += c * s[j - 1].y;
            n.x += w * d[j - 1].x;
            n.y += w * d[j - 1].y;
        }
        a[k].x = m.x + n.y;
        a[k].y = m.y - n.x;
        a[R - k].x = m.x - n.y;
        a[R - k].y = m.y + n.x;
    }
}
// coprime factors: the prime-factor map, no twiddles
template <int N1, int N2, typename C> __device__ __forceinline__ void dft_pfa(C *a) {
    constexpr int N = N1 * N2, E1 = N2 * inv_mod(N2 % N1, N1), E2 = N1 * inv_mod(N1 % N2, N2);
    C t[N2][N1];
#pragma unroll
    for (int i2 = 0; i2 < N2; i2++) {
#pragma unroll
        for (int i1 = 0; i1 < N1; i1++) t[i2][i1] = a[(N2 * i1 + N1 * i2) % N];
        dft<N1>(t[i2]);
    }
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) {
        C b[N2];
#pragma unroll
        for (int i2 = 0; i2 < N2; i2++) b[i2] = t[i2][k1];
        dft<N2>(b);
#pragma unroll
        for (int k2 = 0; k2 < N2; k2++) a[(E1 * k1 + E2 * k2) % N] = b[k2];
    }
}
// N = N1 * N2 with twiddles (9 = 3 x 3, 16 = 4 x 4)
template <int N1, int N2, typename C> __device__ __forceinline__ void dft_ct(C *a) {
    using T = decltype(a[0].x);
    constexpr int N = N1 * N2;
    C t[N2][N1];
#pragma unroll
    for (int i2 = 0; i2 < N2; i2++) {
#pragma unroll
        for (int i1 = 0; i1 < N1; i1++) t[i2][i1] = a[N2 * i1 + i2];
        dft<N1>(t[i2]);
    }
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) {
        C b[N2];
#pragma unroll
        for (int i2 = 0; i2 < N2; i2++) {
            b[i2] = t[i2][k1];
            if (i2 * k1 != 0) {
                C w;
                w.x = (T)cos_r(N, i2 * k1);
                w.y = (T)(-sin_r(N, i2 * k1));
                b[i2] = cmul(b[i2], w);
            }
        }
        dft<N2>(b);
#pragma unroll
        for (int k2 = 0; k2 < N2; k2++) a[k1 + N1 * k2] = b[k2];
    }
}
template <int R, typename C> __device__ __forceinline__ void dft(C *a) {
    if constexpr (R == 2 || R == 3 || R == 4 || R == 5 || R == 8) SmallDFT<R, C>::run(a, -1, nullptr, 0);
    else if constexpr (R == 6) dft_pfa<2, 3>(a);
    else if constexpr (R == 10) dft_pfa<2, 5>(a);
    else if constexpr (R == 12) dft_pfa<3, 4>(a);
    else if constexpr (R == 9) dft_ct<3, 3>(a);
    else if constexpr (R == 16) dft_ct<4, 4>(a);
    else dft_odd<R>(a);
}

template <typename C> __device__ __forceinline__ C swap_ri(C v) {
    C r;
    r.x = v.y;
    r.y = v.x;
    return r;
}

// One stage of radix R over all lines.  The inverse transform is the forward one
// of the values with real and imaginary parts exchanged.
template <int R, bool INV, typename C>
__device__ __forceinline__ void stage(C *buf, const Lines &ln, const Stage &sg, const C *tw) {
    const int total = ln.nl * sg.nbf, m = sg.span, ms = m * ln.es;
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        const int b = fdiv(t, ln.nl_mul), l = t - b * ln.nl;
        const int blk = fdiv(b, sg.span_mul), k1 = b - blk * m;
        C *p = buf + ln.off(l) + (blk * m * R + k1) * ln.es;
        C a[R];
#pragma unroll
        for (int j = 0; j < R; j++) a[j] = INV ? swap_ri(p[j * ms]) : p[j * ms];
        const int e = k1 * sg.twstep;
        if (!INV && e) {
#pragma unroll
            for (int j = 1; j < R; j++) a[j] = cmul(a[j], tw[j * e]);
        }
        dft<R>(a);
        if (INV && e) {
#pragma unroll
            for (int j = 1; j < R; j++) a[j] = cmul(a[j], tw[j * e]);
        }
#pragma unroll
        for (int j = 0; j < R; j++) p[j * ms] = INV ? swap_ri(a[j]) : a[j];
    }
}

// Prime factor above 13.  Chunks of whole butterflies: thread (k, butterfly)
// sums output k of the pair (k, R - k), k = 0 .. (R-1)/2; all threads of a chunk
// have read when the first writes.
template <bool INV, typename C>
__device__ void stage_prime(C *buf, const Lines &ln, const Stage &sg, const C *tw) {
    using T = decltype(buf[0].x);
    const int R = sg.radix, m = sg.span, twstep = sg.twstep, wstep = sg.nbf;
    const unsigned m_mul = sg.span_mul;
    const int nbf = ln.nl * sg.nbf, ms = m * ln.es, H = (R - 1) / 2;
    const int per = blockDim.x / (H + 1) < 1 ? 1 : blockDim.x / (H + 1);
    auto twiddle = [&]() {  // elementwise, over the inputs (forward) or the outputs (inverse)
        if (m == 1) return;
        const int tot = nbf * (R - 1);
        for (int t = threadIdx.x; t < tot; t += blockDim.x) {
            const int j = t / nbf + 1, bf = t - (j - 1) * nbf;
            const int b = fdiv(bf, ln.nl_mul), l = bf - b * ln.nl;
            const int blk = fdiv(b, m_mul), k1 = b - blk * m;
            C *p = buf + ln.off(l) + (blk * m * R + k1 + j * m) * ln.es;
            const C w = tw[j * k1 * twstep];
            *p = INV ? swap_ri(cmul(swap_ri(*p), w)) : cmul(*p, w);
        }
        __syncthreads();
    };
    if (!INV) twiddle();
    for (int c0 = 0; c0 < nbf; c0 += per) {
        const int k = threadIdx.x / per, bf = c0 + (threadIdx.x - k * per);
        const bool on = k <= H && bf < nbf;
        C lo = cmk<C>(0, 0), hi = cmk<C>(0, 0), *p = buf;
        if (on) {
            const int b = fdiv(bf, ln.nl_mul), l = bf - b * ln.nl;
            const int blk = fdiv(b, m_mul), k1 = b - blk * m;
            p = buf + ln.off(l) + (blk * m * R + k1) * ln.es;
            C mm = INV ? swap_ri(p[0]) : p[0], nn = cmk<C>(0, 0);
            int e = 0;  // j * k mod R
#pragma unroll 4
            for (int j = 1; j <= H; j++) {
                e += k;
                if (e >= R) e -= R;
                C u = p[j * ms], v = p[(R - j) * ms];
                if (INV) { u = swap_ri(u); v = swap_ri(v); }
                const C w = tw[e * wstep];  // (cos, -sin)
                const T sx = u.x + v.x, sy = u.y + v.y, dx = u.x - v.x, dy = u.y - v.y;
                mm.x += w.x * sx;
                mm.y += w.x * sy;
                nn.x -= w.y * dx;
                nn.y -= w.y * dy;
            }
            lo.x = mm.x + nn.y;
            lo.y = mm.y - nn.x;
            hi.x = mm.x - nn.y;
            hi.y = mm.y + nn.x;
        }
        __syncthreads();
        if (on) {
            p[k * ms] = INV ? swap_ri(lo) : lo;
            if (k) p[(R - k) * ms] = INV ? swap_ri(hi) : hi;
        }
    }
    __syncthreads();
    if (INV) twiddle();
}

template <bool INV, typename C>
__device__ __noinline__ void run_stage(C *buf, const Lines ln, const Stage sg, const C *tw) {
    switch (sg.radix) {
        case 2: stage<2, INV>(buf, ln, sg, tw); break;
        case 3: stage<3, INV>(buf, ln, sg, tw); break;
        case 4: stage<4, INV>(buf, ln, sg, tw); break;
        case 5: stage<5, INV>(buf, ln, sg, tw); break;
        case 6: stage<6, INV>(buf, ln, sg, tw); break;
        case 7: stage<7, INV>(buf, ln, sg, tw); break;
        case 8: stage<8, INV>(buf, ln, sg, tw); break;
        case 9: stage<9, INV>(buf, ln, sg, tw); break;
        case 10: stage<10, INV>(buf, ln, sg, tw); break;
        case 11: stage<11, INV>(buf, ln, sg, tw); break;
        case 12: stage<12, INV>(buf, ln, sg, tw); break;
        case 13: stage<13, INV>(buf, ln, sg, tw); break;
        case 16: stage<16, INV>(buf, ln, sg, tw); break;
        default: stage_prime<INV>(buf, ln, sg, tw); break;
    }
    __syncthreads();
}

// All stages of an axis over all lines; ends with a block barrier.
template <bool INV, typename C>
__device__ __forceinline__ void transform(C *buf, const Lines ln, const Axis &ap, const C *tw) {
    for (int i = 0; i < ap.nf; i++) run_stage<INV>(buf, ln, ap.st[INV ? i : ap.nf - 1 - i], tw);
}

}  // namespace any
}  // namespace lfts

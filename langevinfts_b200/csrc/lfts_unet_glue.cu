// What stands between the U-Net's convolutions: the channels-last BF16 input,
// average pooling, and upsampling with concatenation, one pass over memory each.
// All are bound by HBM: as torch operations (casts, a mean, three interleaves and
// a concatenation) they took 0.62 of the 1.78 ms of an inference at 64^3, batch 4.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <string>

#include "../../include/lfts_b200.h"

int lfts_internal_fail(const std::string &msg);

namespace {
constexpr int NT = 256;

unsigned blocks_for(long long units) {
    const long long b = (units + NT - 1) / NT;
    return (unsigned)(b < 148 * 16 ? b : 148 * 16);
}
int done() {
    const cudaError_t e = cudaPeekAtLastError();
    return e == cudaSuccess ? 0 : lfts_internal_fail(std::string("unet glue launch: ") + cudaGetErrorString(e));
}

// x [B][cin][P] FP32 -> y [B][P][cpad] BF16, channels past cin zero.  A thread a
// position: reads coalesced along P, writes 16-byte chunks.
__global__ void __launch_bounds__(NT) k_pack_input(const float *__restrict__ x, uint4 *__restrict__ y, long long npos, long long P, int cin,
                                                   int chunks) {
    for (long long t = blockIdx.x * (long long)NT + threadIdx.x; t < npos; t += (long long)gridDim.x * NT) {
        const long long b = t / P, p = t - b * P;
        const float *src = x + b * cin * P + p;
        for (int c = 0; c < chunks; c++) {
            __nv_bfloat162 v[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int ch = c * 8 + 2 * i;
                v[i] = __floats2bfloat162_rn(ch < cin ? src[ch * P] : 0.f, ch + 1 < cin ? src[(ch + 1) * P] : 0.f);
            }
            y[t * chunks + c] = *(uint4 *)v;
        }
    }
}

// mean over 2 x 2 x 2, summed in FP32; a thread an output position and 8 channels
__global__ void __launch_bounds__(NT) k_pool(const uint4 *__restrict__ x, uint4 *__restrict__ y, long long units, int D, int H, int W,
                                             int chunks) {
    for (long long t = blockIdx.x * (long long)NT + threadIdx.x; t < units; t += (long long)gridDim.x * NT) {
        const int c = (int)(t % chunks);
        long long p = t / chunks;
        const int w = (int)(p % W);
        p /= W;
        const int h = (int)(p % H);
        p /= H;  // p = b D + d: input plane 2 p (the input has 2 D planes a batch entry)
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const long long q = ((2 * p + (k >> 2)) * (2 * H) + 2 * h + ((k >> 1) & 1)) * (2 * W) + 2 * w + (k & 1);
            const uint4 v = x[q * chunks + c];
            const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                acc[2 * i] += __uint_as_float(u[i] << 16);
                acc[2 * i + 1] += __uint_as_float(u[i] & 0xFFFF0000u);
            }
        }
        __nv_bfloat162 o[4];
#pragma unroll
        for (int i = 0; i < 4; i++) o[i] = __floats2bfloat162_rn(acc[2 * i] * 0.125f, acc[2 * i + 1] * 0.125f);
        y[t] = *(uint4 *)o;
    }
}

// y = [nearest-neighbour upsampling of a | b]; a thread an output position and 8 channels
__global__ void __launch_bounds__(NT) k_upcat(const uint4 *__restrict__ a, const uint4 *__restrict__ b, uint4 *__restrict__ y,
                                              long long units, int H, int W, int ca, int cb) {
    const int chunks = ca + cb;
    for (long long t = blockIdx.x * (long long)NT + threadIdx.x; t < units; t += (long long)gridDim.x * NT) {
        const int c = (int)(t % chunks);
        const long long p = t / chunks;
        if (c >= ca) {
            y[t] = b[p * cb + c - ca];
            continue;
        }
        const int w = (int)(p % W);
        const long long r = p / W;
        const int h = (int)(r % H);
        const long long d = r / H;  // b D + d with an even D: its half is the coarse plane
        y[t] = a[((d / 2 * (H / 2) + h / 2) * (W / 2) + w / 2) * ca + c];
    }
}
}  // namespace

extern "C" int lfts_unet_pack_input(void *stream, const float *x, void *y, int B, int cin, int D, int H, int W, int cpad) {
    if (!x || !y) return lfts_internal_fail("unet input: null argument");
    if (B < 0 || D < 1 || H < 1 || W < 1 || cin < 1 || cpad < cin || cpad % 8) return lfts_internal_fail("unet input: bad extents or channels");
    if ((uintptr_t)y & 15) return lfts_internal_fail("unet input: the output must be 16-byte aligned");
    const long long P = (long long)D * H * W, n = B * P;
    if (n == 0) return 0;
    k_pack_input<<<blocks_for(n), NT, 0, (cudaStream_t)stream>>>(x, (uint4 *)y, n, P, cin, cpad / 8);
    return done();
}

extern "C" int lfts_unet_pool_bf16(void *stream, const void *x, void *y, int B, int D, int H, int W, int cpad) {
    if (!x || !y) return lfts_internal_fail("unet pool: null argument");
    if (B < 0 || D < 2 || H < 2 || W < 2 || D % 2 || H % 2 || W % 2 || cpad < 8 || cpad % 8)
        return lfts_internal_fail("unet pool: extents must be even and channels a multiple of 8");
    if (((uintptr_t)x | (uintptr_t)y) & 15) return lfts_internal_fail("unet pool: buffers must be 16-byte aligned");
    const long long units = (long long)B * (D / 2) * (H / 2) * (W / 2) * (cpad / 8);
    if (units == 0) return 0;
    k_pool<<<blocks_for(units), NT, 0, (cudaStream_t)stream>>>((const uint4 *)x, (uint4 *)y, units, D / 2, H / 2, W / 2, cpad / 8);
    return done();
}

extern "C" int lfts_unet_upcat_bf16(void *stream, const void *a, const void *b, void *y, int B, int D, int H, int W, int ca, int cb) {
    if (!a || !b || !y) return lfts_internal_fail("unet upcat: null argument");
    if (B < 0 || D < 2 || H < 2 || W < 2 || D % 2 || H % 2 || W % 2 || ca < 8 || cb < 8 || ca % 8 || cb % 8)
        return lfts_internal_fail("unet upcat: extents must be even and channels multiples of 8");
    if (((uintptr_t)a | (uintptr_t)b | (uintptr_t)y) & 15) return lfts_internal_fail("unet upcat: buffers must be 16-byte aligned");
    const long long units = (long long)B * D * H * W * ((ca + cb) / 8);
    if (units == 0) return 0;
    k_upcat<<<blocks_for(units), NT, 0, (cudaStream_t)stream>>>((const uint4 *)a, (const uint4 *)b, (uint4 *)y, units, H, W, ca / 8, cb / 8);
    return done();
}

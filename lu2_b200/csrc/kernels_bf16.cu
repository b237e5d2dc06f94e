// kernels_bf16.cu -- FP32 -> BF16 conversion of the precision form's L21
// panel (with its per-panel power-of-two scale) for the tcgen05 trailing
// update in kernels_lowp.cu.
#include <cuda_bf16.h>

#include "lu2gpu_internal.cuh"

namespace lu2gpu {

// ---------------------------------------------------------------------------
// FP32 <-> BF16 helpers for the precision form

// out (rows x cols, stride ldo, BF16) = in (FP32, stride ldi) * *scale
// A warp takes 128 columns of a row at a time, four such pieces in flight
// (element by element, with a 64-bit division each, 7.4 us a panel of 256
// columns on average in a solve of order 12288; here 3.0).
__global__ void __launch_bounds__(256) f32_to_bf16_kernel(const float *__restrict__ in, long ldi,
                                                          __nv_bfloat16 *__restrict__ out, long ldo, int rows, int cols,
                                                          const float *scalep)
{
    const float scale = *scalep;
    const int lane = threadIdx.x & 31, segs = (cols + 127) / 128, step = gridDim.x * 8;
    const bool vec = (reinterpret_cast<uintptr_t>(in) & 15) == 0 && (ldi & 3) == 0 &&
                     (reinterpret_cast<uintptr_t>(out) & 7) == 0 && (ldo & 3) == 0;
    for (long u0 = blockIdx.x * 8 + (threadIdx.x >> 5); u0 < (long)rows * segs; u0 += 4 * step) {
        float v[4][4];
        size_t at[4];
        int have[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const long u = u0 + (long)q * step;
            const int r = (int)((unsigned)u / (unsigned)segs), c = (int)(u - (long)r * segs) * 128 + 4 * lane;
            const float *p = in + (size_t)r * ldi + c;
            at[q] = (size_t)r * ldo + c;
            have[q] = u < (long)rows * segs ? min(4, cols - c) : 0;
            if (vec && have[q] == 4) {
                const float4 w = *reinterpret_cast<const float4 *>(p);
                v[q][0] = w.x;
                v[q][1] = w.y;
                v[q][2] = w.z;
                v[q][3] = w.w;
            } else {
#pragma unroll
                for (int e = 0; e < 4; e++) v[q][e] = e < have[q] ? p[e] : 0.f;
            }
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (vec && have[q] == 4) {
                __nv_bfloat162 w[2];
                w[0].x = __float2bfloat16_rn(v[q][0] * scale);
                w[0].y = __float2bfloat16_rn(v[q][1] * scale);
                w[1].x = __float2bfloat16_rn(v[q][2] * scale);
                w[1].y = __float2bfloat16_rn(v[q][3] * scale);
                *reinterpret_cast<uint2 *>(out + at[q]) = *reinterpret_cast<uint2 *>(w);
            } else {
#pragma unroll
                for (int e = 0; e < 4; e++)
                    if (e < have[q]) out[at[q] + e] = __float2bfloat16_rn(v[q][e] * scale);
            }
        }
    }
}

cudaError_t launch_f32_to_bf16(const float *in, long ldi, void *out, long ldo, int rows, int cols,
                               const float *scale, cudaStream_t st)
{
    if (rows <= 0 || cols <= 0) return cudaSuccess;
    const long units = (long)rows * ((cols + 127) / 128);
    const long blocks = units < 148 * 8 * 32 ? (units + 31) / 32 : 148 * 8;
    count_launch();
    f32_to_bf16_kernel<<<(unsigned)blocks, 256, 0, st>>>(in, ldi, (__nv_bfloat16 *)out, ldo, rows, cols, scale);
    return cudaGetLastError();
}

}  // namespace lu2gpu

// kernels_mixed.cu -- support kernels of the precision form: the FP32 updates
// inside the panel recursion, the per-panel power-of-two scales of the BF16
// operands, FP64 <-> FP32 conversions, the FP64 residual of the iterative
// refinement and the per-panel update of the FP32 forward solve.
#include <algorithm>

#include <cuda_bf16.h>

#include "lu2gpu_internal.cuh"

namespace lu2gpu {

// ---------------------------------------------------------------------------
// C -= A Bt^T in FP32 on the CUDA cores (exact FP32 arithmetic for the panel,
// which the precision form keeps in FP32).  64 x 64 tiles, 256 threads of 4 x 4,
// each sum over k from zero and subtracted once.
// These updates have K = 64 or 128 and a few hundred tiles, so that the trips
// to memory bound them: C is read before the products, the next 32 columns of
// A and Bt beside them (16-byte loads where VEC: rows 16-byte aligned, K a
// multiple of 4), two buffers in shared memory.  The operands lie there k-major
// with row r of column k at r ^ 4 (k / 4), which puts a warp's transposing
// stores on distinct banks and keeps four rows together.
// One slab at a time, read value by value and C last -> this: M = 4000, N = K =
// 64 9.6 -> 5.0 us, N = K = 128 15.4 -> 8.5; M = 12000, 128 22.4 -> 16.7.
constexpr int SG_T = 64, SG_K = 32;

template <bool VEC>
__global__ void __launch_bounds__(256) sgemm_update_kernel(const float *__restrict__ a, long lda,
                                                           const float *__restrict__ bt, float *c, long ldc, int M,
                                                           int N, int K)
{
    __shared__ __align__(16) float As[2][SG_K * SG_T], Bs[2][SG_K * SG_T];
    const int m0 = blockIdx.x * SG_T, n0 = blockIdx.y * SG_T, tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    // this thread's C: rows m0 + 4 ty + i, columns n0 + 4 tx + j
    const bool cvec = VEC && n0 + SG_T <= N && (ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(c) & 15) == 0;
    float *cp = c + (size_t)(m0 + 4 * ty) * ldc + n0 + 4 * tx;
    float old[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if (cvec && m0 + 4 * ty + i < M) {
            const float4 v = *reinterpret_cast<const float4 *>(cp + (size_t)i * ldc);
            old[i][0] = v.x;
            old[i][1] = v.y;
            old[i][2] = v.z;
            old[i][3] = v.w;
        } else {
#pragma unroll
            for (int j = 0; j < 4; j++)
                old[i][j] = m0 + 4 * ty + i < M && n0 + 4 * tx + j < N ? cp[(size_t)i * ldc + j] : 0.f;
        }
    }
    // this thread's part of a slab: rows tid / 8 and + 32, columns 4 (tid % 8) ..
    const int sr = tid >> 3, sk = 4 * (tid & 7);
    float4 ra[2], rb[2];
    auto fetch = [&](const float *p, long ld, int row0, int rows, int k0, float4 (&v)[2]) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int r = row0 + sr + 32 * h, k = k0 + sk;
            const float *q = p + (size_t)r * ld + k;
            if (VEC)
                v[h] = r < rows && k < K ? *reinterpret_cast<const float4 *>(q) : make_float4(0.f, 0.f, 0.f, 0.f);
            else
                v[h] = make_float4(r < rows && k < K ? q[0] : 0.f, r < rows && k + 1 < K ? q[1] : 0.f,
                                   r < rows && k + 2 < K ? q[2] : 0.f, r < rows && k + 3 < K ? q[3] : 0.f);
        }
    };
    auto load = [&](int k0) {
        fetch(a, lda, m0, M, k0, ra);
        fetch(bt, K, n0, N, k0, rb);
    };
    auto store = [&](int buf) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int r = (sr + 32 * h) ^ sk;
            float *pa = As[buf] + sk * SG_T + r, *pb = Bs[buf] + sk * SG_T + r;
            pa[0] = ra[h].x;
            pa[SG_T] = ra[h].y;
            pa[2 * SG_T] = ra[h].z;
            pa[3 * SG_T] = ra[h].w;
            pb[0] = rb[h].x;
            pb[SG_T] = rb[h].y;
            pb[2 * SG_T] = rb[h].z;
            pb[3 * SG_T] = rb[h].w;
        }
    };
    float acc[4][4] = {};
    load(0);
    store(0);
    __syncthreads();
    for (int k0 = 0, buf = 0; k0 < K; k0 += SG_K, buf ^= 1) {
        const bool more = k0 + SG_K < K;
        if (more) load(k0 + SG_K);
#pragma unroll 8
        for (int k = 0; k < SG_K; k++) {
            const int sw = k & ~3;
            const float4 av = *reinterpret_cast<const float4 *>(As[buf] + k * SG_T + ((4 * ty) ^ sw));
            const float4 bv = *reinterpret_cast<const float4 *>(Bs[buf] + k * SG_T + ((4 * tx) ^ sw));
            const float x[4] = {av.x, av.y, av.z, av.w}, y[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(x[i], y[j], acc[i][j]);
        }
        if (more) store(buf ^ 1);
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if (m0 + 4 * ty + i >= M) continue;
        if (cvec) {
            *reinterpret_cast<float4 *>(cp + (size_t)i * ldc) = make_float4(
                old[i][0] - acc[i][0], old[i][1] - acc[i][1], old[i][2] - acc[i][2], old[i][3] - acc[i][3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (n0 + 4 * tx + j < N) cp[(size_t)i * ldc + j] = old[i][j] - acc[i][j];
        }
    }
}

cudaError_t launch_sgemm_update(const float *a, long lda, const float *bt, float *c, long ldc, int M, int N, int K,
                                cudaStream_t st)
{
    if (M <= 0 || N <= 0 || K <= 0) return cudaSuccess;
    dim3 grid((M + SG_T - 1) / SG_T, (N + SG_T - 1) / SG_T);
    if (grid.y > 65535) return cudaErrorInvalidConfiguration;
    count_launch();
    const bool vec = (reinterpret_cast<uintptr_t>(a) & 15) == 0 && (lda & 3) == 0 &&
                     (reinterpret_cast<uintptr_t>(bt) & 15) == 0 && (K & 3) == 0;
    if (vec)
        sgemm_update_kernel<true><<<grid, 256, 0, st>>>(a, lda, bt, c, ldc, M, N, K);
    else
        sgemm_update_kernel<false><<<grid, 256, 0, st>>>(a, lda, bt, c, ldc, M, N, K);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// per-panel power-of-two scales

// amax_bits[i] = max(amax_bits[i], max |x|) of the two operands of an update in
// one launch (non-negative floats order as their bits).  A warp takes 128
// columns of a row at a time, four such pieces in flight.  (One element per
// thread and step, with a 64-bit division each: 9.7 us an operand on average in
// a solve of order 12288, here 3.7 for both.)
struct AbsmaxArgs {
    const float *x[2];
    long ld[2];
    int rows[2], cols[2];
};

__global__ void __launch_bounds__(256) absmax2_kernel(const AbsmaxArgs P, unsigned *amax_bits)
{
    const int which = blockIdx.y, lane = threadIdx.x & 31;
    const float *x = which ? P.x[1] : P.x[0];
    const long ld = which ? P.ld[1] : P.ld[0];
    const int rows = which ? P.rows[1] : P.rows[0], cols = which ? P.cols[1] : P.cols[0], segs = (cols + 127) / 128;
    const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0 && (ld & 3) == 0;
    const int step = gridDim.x * 8;
    float m = 0.f;
    for (long u0 = blockIdx.x * 8 + (threadIdx.x >> 5); u0 < (long)rows * segs; u0 += 4 * step) {
        float4 v[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const long u = u0 + (long)q * step;
            v[q] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (u < (long)rows * segs) {
                const int r = (int)((unsigned)u / (unsigned)segs), c = (int)(u - (long)r * segs) * 128 + 4 * lane;
                const float *p = x + (size_t)r * ld + c;
                if (vec && c + 3 < cols) {
                    v[q] = *reinterpret_cast<const float4 *>(p);
                } else {
                    if (c < cols) v[q].x = p[0];
                    if (c + 1 < cols) v[q].y = p[1];
                    if (c + 2 < cols) v[q].z = p[2];
                    if (c + 3 < cols) v[q].w = p[3];
                }
            }
        }
#pragma unroll
        for (int q = 0; q < 4; q++)
            m = fmaxf(fmaxf(fmaxf(m, fabsf(v[q].x)), fmaxf(fabsf(v[q].y), fabsf(v[q].z))), fabsf(v[q].w));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ unsigned warp_max[8];
    if (lane == 0) warp_max[threadIdx.x >> 5] = __float_as_uint(m);
    __syncthreads();
    if (threadIdx.x < 8) {
        const unsigned b = __reduce_max_sync(0xffu, warp_max[threadIdx.x]);
        if (threadIdx.x == 0) atomicMax(&amax_bits[which], b);
    }
}

cudaError_t launch_absmax2(const float *x0, long ld0, int rows0, int cols0, const float *x1, long ld1, int rows1,
                           int cols1, unsigned *amax_bits, cudaStream_t st)
{
    if (rows0 <= 0 || cols0 <= 0 || rows1 <= 0 || cols1 <= 0) return cudaErrorInvalidValue;
    const AbsmaxArgs P{{x0, x1}, {ld0, ld1}, {rows0, rows1}, {cols0, cols1}};
    const long units = std::max((long)rows0 * ((cols0 + 127) / 128), (long)rows1 * ((cols1 + 127) / 128));
    count_launch();
    absmax2_kernel<<<dim3((unsigned)std::min(148L * 4, (units + 31) / 32), 2), 256, 0, st>>>(P, amax_bits);
    return cudaGetLastError();
}

// scales[0] = 1/sL, scales[1] = 1/sU, scales[2] = sL*sU for the two maxima in
// amax_bits[0..1]; sX = 2^e with max|X| <= 2^e (1 for an all-zero block).
__global__ void panel_scales_kernel(const unsigned *amax_bits, float *scales)
{
    float s[2];
    for (int i = 0; i < 2; i++) {
        const float m = __uint_as_float(amax_bits[i]);
        int e = 0;
        if (m > 0.f && isfinite(m)) frexpf(m, &e);
        s[i] = ldexpf(1.f, e);
    }
    scales[0] = 1.f / s[0];
    scales[1] = 1.f / s[1];
    scales[2] = s[0] * s[1];
}

cudaError_t launch_panel_scales(const unsigned *amax_bits, float *scales, cudaStream_t st)
{
    count_launch();
    panel_scales_kernel<<<1, 1, 0, st>>>(amax_bits, scales);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// conversions

__global__ void f64_to_f32_kernel(const double *__restrict__ x, long ldx, float *__restrict__ y, long ldy, int rows,
                                  int cols)
{
    const long total = (long)rows * cols;
    for (long idx = (long)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (long)gridDim.x * blockDim.x) {
        const long r = idx / cols, c = idx - r * cols;
        y[r * ldy + c] = (float)x[r * ldx + c];
    }
}

__global__ void f32_to_f64_kernel(const float *__restrict__ x, long ldx, double *__restrict__ y, long ldy, int rows,
                                  int cols)
{
    const long total = (long)rows * cols;
    for (long idx = (long)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (long)gridDim.x * blockDim.x) {
        const long r = idx / cols, c = idx - r * cols;
        y[r * ldy + c] = (double)x[r * ldx + c];
    }
}

static unsigned grid_for(long total)
{
    long b = (total + 255) / 256;
    if (b > 148 * 32) b = 148 * 32;
    return (unsigned)(b > 0 ? b : 1);
}

cudaError_t launch_f64_to_f32(const double *x, long ldx, float *y, long ldy, int rows, int cols, cudaStream_t st)
{
    if (rows <= 0 || cols <= 0) return cudaSuccess;
    count_launch();
    f64_to_f32_kernel<<<grid_for((long)rows * cols), 256, 0, st>>>(x, ldx, y, ldy, rows, cols);
    return cudaGetLastError();
}

cudaError_t launch_f32_to_f64(const float *x, long ldx, double *y, long ldy, int rows, int cols, cudaStream_t st)
{
    if (rows <= 0 || cols <= 0) return cudaSuccess;
    count_launch();
    f32_to_f64_kernel<<<grid_for((long)rows * cols), 256, 0, st>>>(x, ldx, y, ldy, rows, cols);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// r = b - A x in FP64, one warp per row (the refinement's residual; reads A once)
__global__ void __launch_bounds__(256) residual_kernel(const double *__restrict__ a, long lda, int n,
                                                       const double *__restrict__ b, const double *__restrict__ x,
                                                       double *__restrict__ r, double *__restrict__ rowabs)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = blockIdx.x * 8 + warp; i < n; i += gridDim.x * 8) {
        const double *row = a + (size_t)i * lda;
        double s = 0.0, sa = 0.0;
        for (int j = lane * 2; j < n; j += 64) {
            if (j + 1 < n) {
                const double2 v = __ldcs(reinterpret_cast<const double2 *>(row + j));
                s = fma(v.x, x[j], s);
                s = fma(v.y, x[j + 1], s);
                sa += fabs(v.x) + fabs(v.y);
            } else {
                const double v = __ldcs(row + j);
                s = fma(v, x[j], s);
                sa += fabs(v);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            s += __shfl_xor_sync(0xffffffffu, s, o);
            sa += __shfl_xor_sync(0xffffffffu, sa, o);
        }
        if (lane == 0) {
            r[i] = b ? b[i] - s : s;  // without b: the product A x
            if (rowabs) rowabs[i] = sa;
        }
    }
}

cudaError_t launch_residual(const double *a, long lda, int n, const double *b, const double *x, double *r,
                            double *rowabs, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    if ((lda & 1) || (reinterpret_cast<uintptr_t>(a) & 15)) return cudaErrorInvalidValue;
    int blocks = (n + 7) / 8;
    if (blocks > 148 * 16) blocks = 148 * 16;
    count_launch();
    residual_kernel<<<blocks, 256, 0, st>>>(a, lda, n, b, x, r, rowabs);
    return cudaGetLastError();
}

// y[i] -= sum_k l[i][k] v[k] for i < rows, K <= 512 (one warp per row)
__global__ void __launch_bounds__(256) gemv_sub_kernel(const float *__restrict__ l, long ld, int rows, int K,
                                                       const float *__restrict__ v, float *__restrict__ y)
{
    __shared__ float vs[512];
    for (int k = threadIdx.x; k < K; k += blockDim.x) vs[k] = v[k];
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = blockIdx.x * 8 + warp; i < rows; i += gridDim.x * 8) {
        const float *row = l + (size_t)i * ld;
        float s = 0.f;
        for (int k = lane; k < K; k += 32) s = fmaf(__ldcs(row + k), vs[k], s);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) y[i] -= s;
    }
}

cudaError_t launch_gemv_sub(const float *l, long ld, int rows, int K, const float *v, float *y, cudaStream_t st)
{
    if (rows <= 0 || K <= 0) return cudaSuccess;
    if (K > 512) return cudaErrorInvalidValue;
    int blocks = (rows + 7) / 8;
    if (blocks > 148 * 16) blocks = 148 * 16;
    count_launch();
    gemv_sub_kernel<<<blocks, 256, 0, st>>>(l, ld, rows, K, v, y);
    return cudaGetLastError();
}

// bt[j][k] = BF16(u[k][j] * *scale): the U block row (K x N FP32, stride ld)
// transposed into the K-contiguous B operand of the BF16 update
__global__ void f32_transpose_bf16_kernel(const float *__restrict__ u, long ld, int K, int N,
                                          __nv_bfloat16 *__restrict__ bt, const float *__restrict__ scalep)
{
    __shared__ float tile[32][33];
    const float scale = *scalep;
    const int j0 = blockIdx.x * 32, k0 = blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int k = k0 + r, j = j0 + threadIdx.x;
        tile[r][threadIdx.x] = (k < K && j < N) ? u[(size_t)k * ld + j] : 0.f;
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int j = j0 + r, k = k0 + threadIdx.x;
        if (j < N && k < K) bt[(size_t)j * K + k] = __float2bfloat16_rn(tile[threadIdx.x][r] * scale);
    }
}

cudaError_t launch_f32_transpose_bf16(const float *u, long ld, int K, int N, void *bt, const float *scale,
                                      cudaStream_t st)
{
    if (K <= 0 || N <= 0) return cudaSuccess;
    dim3 grid((N + 31) / 32, (K + 31) / 32);
    count_launch();
    f32_transpose_bf16_kernel<<<grid, dim3(32, 8), 0, st>>>(u, ld, K, N, (__nv_bfloat16 *)bt, scale);
    return cudaGetLastError();
}

// x[i] += (double)d[i]
__global__ void add_f32_to_f64_kernel(const float *__restrict__ d, double *__restrict__ x, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) x[i] += (double)d[i];
}

cudaError_t launch_add_f32_to_f64(const float *d, double *x, int n, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    count_launch();
    add_f32_to_f64_kernel<<<grid_for(n), 256, 0, st>>>(d, x, n);
    return cudaGetLastError();
}

// out[slot] = max_i |v[i]| for a double vector (out zeroed by the caller;
// non-negative doubles order as their bits)
__global__ void vec_absmax_kernel(const double *__restrict__ v, int n, unsigned long long *out)
{
    double m = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) m = fmax(m, fabs(v[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, (unsigned long long)__double_as_longlong(m));
}

cudaError_t launch_vec_absmax(const double *v, int n, unsigned long long *out, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    count_launch();
    vec_absmax_kernel<<<grid_for(n) < 296 ? grid_for(n) : 296, 256, 0, st>>>(v, n, out);
    return cudaGetLastError();
}

}  // namespace lu2gpu

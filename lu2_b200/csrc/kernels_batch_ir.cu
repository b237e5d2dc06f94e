// kernels_batch_ir.cu -- the batching form's FP32-LU + FP64 iterative
// refinement variant: every system's FP64 augmented matrix (left unchanged
// until x is written into its b columns) is converted to FP32, factored in
// FP32, and refined in FP64 -- r = b - A x from the FP64 matrix, the
// correction solved with the FP32 factors -- until every right-hand side has
// an HPL scaled residual below 16 however it is summed (or max_iter corrections).
//
// Factor storage follows lu2's elimination (lu2.c:541-554, lu2tlib.c:1057-
// 1059): the pivot row is scaled by 1/pivot right of the diagonal (a unit
// upper U'), the columns below keep the unscaled multipliers times the pivot
// (L' lower with the pivots on its diagonal).  Unlike lu2, whose solve rides
// along as augmented columns, the refinement needs the factors for new
// right-hand sides, so rows are exchanged over their full width (LAPACK
// order): P A = L' U', solved as y = L'^{-1} P r, d = U'^{-1} y.
//
// What bounds it is the chain of one system: the pivot search and row step of
// each column, and in the solves the substitution inside a block of 32 rows.
// The exchanges are kept as one permutation (original row of each final row),
// so that a right-hand side is permuted by one gather instead of n dependent
// swaps; the solves hold their diagonal block in registers; the panel's right
// part with 16 columns and the 8 x 4 tiles of the update stay in registers.
// 1000 systems, best of the launch shapes, before -> after: n in [16, 63]
// 0.56 -> 0.29 ms, [64, 127] 2.00 -> 1.13, [128, 255] 6.87 -> 3.56, [256, 512]
// 24.9 -> 13.0 ms.
//
// One CTA per system from a largest-first queue, as in the FP64 variant.
// Systems whose FP32 matrix fits shared memory are factored and solved
// there; larger ones are factored blocked in their FP32 slot of the work
// arena (panel of pw columns in shared memory) and solved from it.
#include <climits>

#include "lu2gpu_internal.cuh"

namespace lu2gpu {

// FP32 factorization of F (n x n, stride fs) held in shared memory: per
// column warp 0 alone (warp-synchronously) searches the pivot, exchanges the
// full rows and scales the pivot row, then after one barrier every thread
// takes part in the rank-1 update -- two barriers per column
__device__ void ir_factor_smem(float *F, int n, int fs, int *perm, int *first_zero)
{
    const int T = blockDim.x, tid = threadIdx.x;
    for (int k = 0; k < n; k++) {
        if (tid < 32) {
            const int lane = tid;
            float v = -1.f;
            int p = INT_MAX;
            for (int r = k + lane; r < n; r += 32) {
                const float a = fabsf(F[r * fs + k]);
                if (a > v) {
                    v = a;
                    p = r;
                }
            }
            warp_argmax_redux(v, p);
            if (p == INT_MAX) p = k;
            if (lane == 0 && p != k) {
                const int t = perm[k];
                perm[k] = perm[p];
                perm[p] = t;
            }
            if (p != k)
                for (int c = lane; c < n; c += 32) {
                    const float t = F[k * fs + c];
                    F[k * fs + c] = F[p * fs + c];
                    F[p * fs + c] = t;
                }
            __syncwarp();
            const float d = F[k * fs + k];
            __syncwarp();  // every lane has read the pivot before the row is scaled
            if (d != 0.f) {
                const float inv = 1.f / d;
                for (int c = k + 1 + lane; c < n; c += 32) F[k * fs + c] *= inv;
            } else if (lane == 0 && !*first_zero) {
                *first_zero = k + 1;
            }
        }
        __syncthreads();
        if (F[k * fs + k] == 0.f) continue;  // (uniform: every thread reads the same pivot)
        // a warp per row (no division of a running index), lanes over its columns
        for (int r = k + 1 + (tid >> 5); r < n; r += T >> 5) {
            const float l = F[r * fs + k];
            for (int c = k + 1 + (tid & 31); c < n; c += 32) F[r * fs + c] -= l * F[k * fs + c];
        }
        __syncthreads();
    }
}

// A panel's composed exchanges on the columns left of it (full-width rows)
// and, with the unit-lower solve and the 1/pivot scaling, on the right part,
// one thread per column: every gather first (16 loads in flight), then the
// displaced rows (read before the rows they come from are rewritten, written
// after every gather, since a gathered row may be one of them), then the
// panel's rows.  WM = 16: a 16-column panel, whose 16 values stay in registers.
template <int WM>
__device__ __forceinline__ void ir_right(float *F, int n, int k0, int cs, int ne, const float *P, int ps,
                                         const float *dinv, const BatchPlan &plan, int w)
{
    const int nleft = k0, ncols = k0 + (n - cs), T = blockDim.x;
    for (int jj = threadIdx.x; jj < ncols; jj += T) {
        const int j = jj < nleft ? jj : cs + (jj - nleft);
        float x[WM];
        for (int q0 = 0; q0 < (WM == 16 ? 16 : w); q0 += 16) {
            float v[16];
#pragma unroll
            for (int u = 0; u < 16; u++) v[u] = q0 + u < w ? F[(size_t)(k0 + plan.blk[q0 + u]) * n + j] : 0.f;
#pragma unroll
            for (int u = 0; u < 16; u++)
                if (q0 + u < w) x[q0 + u] = v[u];
        }
        for (int e0 = 0; e0 < ne; e0 += 16) {
            float v[16];
#pragma unroll
            for (int u = 0; u < 16; u++) v[u] = e0 + u < ne ? F[(size_t)(k0 + plan.ext_src[e0 + u]) * n + j] : 0.f;
#pragma unroll
            for (int u = 0; u < 16; u++)
                if (e0 + u < ne) F[(size_t)(k0 + plan.ext_row[e0 + u]) * n + j] = v[u];
        }
        if constexpr (WM == 16) {
            if (jj >= nleft)
#pragma unroll
                for (int r = 0; r < 16; r++) {
                    float s = x[r];
#pragma unroll
                    for (int l = 0; l < r; l++) s -= P[r * ps + l] * x[l];
                    x[r] = s * dinv[r];
                }
#pragma unroll
            for (int c = 0; c < 16; c++) F[(size_t)(k0 + c) * n + j] = x[c];
        } else {
            if (jj >= nleft)
                for (int r = 0; r < w; r++) {
                    float s = x[r];
                    for (int l = 0; l < r; l++) s -= P[r * ps + l] * x[l];
                    x[r] = s * dinv[r];
                }
            for (int c = 0; c < w; c++) F[(size_t)(k0 + c) * n + j] = x[c];
        }
    }
}

// FP32 factorization of F (n x n, stride n) in global memory, panel of pw
// columns staged in shared memory (U: pw x 64, 16-byte aligned, then P: rows x
// (pw+1)).  The panel is factored by the first NWP warps (up to 4), thread pt
// owning the panel rows c + pt + k S (S = 32 NWP) for both the pivot search of
// column c and the rank-1 step of column c - 1, with two named barriers of the
// S threads per column; warp 0 composes the panel's row exchanges into one
// plan, which the columns left of the panel (full-width exchanges) and the
// right part then apply with independent loads instead of one dependent swap
// per pivot, and which moves the original row numbers (perm) along.
__device__ void ir_factor_blocked(float *F, int n, int pw, float *P, float *U, int *perm, float *dinv,
                                  int *first_zero, float *s_v, int *s_i, BatchPlan &plan)
{
    const int T = blockDim.x, tid = threadIdx.x;
    const int ps = pw + 1;  // odd panel row stride: a column's rows fall in distinct banks
    for (int k0 = 0; k0 < n; k0 += pw) {
        const int w = min(pw, n - k0), rows = n - k0;
        for (int idx = tid; idx < rows * w; idx += T) {
            const int r = idx / w, c = idx - r * w;
            P[r * ps + c] = F[(size_t)(k0 + r) * n + k0 + c];
        }
        __syncthreads();
        const int nwp = min(4, T >> 5), S = 32 * nwp;
        if (tid < S) {
            const int lane = tid & 31, pw_ = tid >> 5;
            if (tid < 32) {
                for (int q = lane; q < w; q += 32) plan.blk[q] = q;
                if (lane == 0) plan.next = 0;
                __syncwarp();
            }
            for (int c = 0; c < w; c++) {
                float v = -1.f;
                int p = INT_MAX;
                for (int r = c + tid; r < rows; r += S) {
                    const float a = fabsf(P[r * ps + c]);
                    if (a > v) {
                        v = a;
                        p = r;
                    }
                }
                if (lane == warp_argmax_redux(v, p)) {
                    s_v[pw_] = v;
                    s_i[pw_] = p;
                }
                asm volatile("bar.sync 1, %0;" ::"r"(S) : "memory");
                v = s_v[0];
                p = s_i[0];
                for (int q = 1; q < nwp; q++)
                    if (s_v[q] > v || (s_v[q] == v && s_i[q] < p)) {
                        v = s_v[q];
                        p = s_i[q];
                    }
                if (p == INT_MAX) p = c;
                if (tid < 32) {
                    if (p != c)
                        for (int j = lane; j < w; j += 32) {
                            const float t = P[c * ps + j];
                            P[c * ps + j] = P[p * ps + j];
                            P[p * ps + j] = t;
                        }
                    __syncwarp();
                    const float d = P[c * ps + c];
                    const bool zero = (d == 0.f);
                    const float inv = zero ? 1.f : 1.f / d;
                    if (lane == 0) dinv[c] = inv;
                    __syncwarp();  // every lane has read the pivot before the row is scaled
                    if (!zero)
                        for (int j = c + 1 + lane; j < w; j += 32) P[c * ps + j] *= inv;
                    batch_plan_step(plan, c, p, w, lane);
                }
                asm volatile("bar.sync 1, %0;" ::"r"(S) : "memory");
                const bool zero = (P[c * ps + c] == 0.f);
                if (zero && tid == 0 && !*first_zero) *first_zero = k0 + c + 1;
                if (!zero)
                    for (int r = c + 1 + tid; r < rows; r += S) {
                        const float l = P[r * ps + c];
                        for (int j = c + 1; j < w; j++) P[r * ps + j] -= l * P[c * ps + j];
                    }
            }
        }
        __syncthreads();
        for (int idx = tid; idx < rows * w; idx += T) {
            const int r = idx / w, c = idx - r * w;
            F[(size_t)(k0 + r) * n + k0 + c] = P[r * ps + c];
        }
        const int cs = k0 + w, ne = plan.next;
        if (tid < 64) {  // and to the rows' original numbers (w <= 64 panel rows, as many displaced)
            const int q = tid < w ? perm[k0 + plan.blk[tid]] : 0, e = tid < ne ? perm[k0 + plan.ext_src[tid]] : 0;
            asm volatile("bar.sync 2, 64;" ::: "memory");
            if (tid < w) perm[k0 + tid] = q;
            if (tid < ne) perm[k0 + plan.ext_row[tid]] = e;
        }
        if (w == 16)
            ir_right<16>(F, n, k0, cs, ne, P, ps, dinv, plan, 16);
        else
            ir_right<64>(F, n, k0, cs, ne, P, ps, dinv, plan, w);
        __syncthreads();
        // trailing update F[cs.., cs..] -= L21 U12 in 64-column chunks
        const int h = n - cs;
        for (int c0 = cs; c0 < n && h > 0; c0 += 64) {
            const int cw = min(64, n - c0);
            for (int idx = tid; idx < w * 64; idx += T) {
                const int l = idx >> 6, c = idx & 63;
                U[l * 64 + c] = (c < cw) ? F[(size_t)(k0 + l) * n + c0 + c] : 0.f;
            }
            __syncthreads();
            // 8 x 4 per thread: the chunk's row by 16-byte loads, the panel's
            // multipliers as broadcasts (4 x 4 with scalar loads read 8 values
            // for 16 products; with the right part of 16-column panels in
            // registers [256, 512] went from 16.7 to 13.0 ms)
            const int tx = tid & 15, ty = tid >> 4, tys = T >> 4;
            for (int rb = ty * 8; rb < h; rb += tys * 8) {
                float acc[8][4] = {};
                const float *lp = P + (size_t)(w + rb) * ps;
                const int last = h - 1 - rb;  // rows past the matrix repeat its last
#pragma unroll 4
                for (int l = 0; l < w; l++) {
                    const float4 bv = *reinterpret_cast<const float4 *>(U + l * 64 + tx * 4);
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const float av = lp[min(i, last) * ps + l];
                        acc[i][0] = fmaf(av, bv.x, acc[i][0]);
                        acc[i][1] = fmaf(av, bv.y, acc[i][1]);
                        acc[i][2] = fmaf(av, bv.z, acc[i][2]);
                        acc[i][3] = fmaf(av, bv.w, acc[i][3]);
                    }
                }
                float *row = F + (size_t)(cs + rb) * n + c0 + tx * 4;
                float old[8][4];
#pragma unroll
                for (int i = 0; i < 8; i++)
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        old[i][q] = rb + i < h && tx * 4 + q < cw ? row[(size_t)i * n + q] : 0.f;
#pragma unroll
                for (int i = 0; i < 8; i++)
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        if (rb + i < h && tx * 4 + q < cw) row[(size_t)i * n + q] = old[i][q] - acc[i][q];
            }
            __syncthreads();
        }
    }
}

// V (r vectors of n, one after the other, shared memory) := U'^{-1} L'^{-1} V
// with the FP32 factors F (stride fs, shared or global memory), V permuted by
// the caller.  Blocks of 32 rows: one warp per right-hand side solves the
// diagonal block, a row per lane in registers (loaded before the barrier that
// its turn waits for) and the diagonal's reciprocals once, then every thread
// updates rows beyond it.  (With the block read column by column inside the
// substitution each step waited for memory and a division.)
__device__ void ir_solve(const float *F, int n, int fs, float *V, int r)
{
    const int T = blockDim.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = T >> 5;
    float f[32];
    // row b0 + lane of the diagonal block
    auto fetch = [&](int b0, int bw) {
        const float *row = F + (size_t)(b0 + min(lane, bw - 1)) * fs + b0;
#pragma unroll
        for (int k = 0; k < 32; k++) f[k] = k < bw ? row[k] : 0.f;
    };
    auto update = [&](int i0, int i1, int b0, int bw) {
        for (int idx = tid; idx < (i1 - i0) * r; idx += T) {
            const int i = i0 + (r == 1 ? idx : idx / r), q = r == 1 ? 0 : idx % r;
            const float *row = F + (size_t)i * fs + b0, *v = V + (size_t)q * n + b0;
            float s0 = 0.f, s1 = 0.f;
            if (bw == 32) {
#pragma unroll
                for (int k = 0; k < 32; k += 2) {
                    s0 = fmaf(row[k], v[k], s0);
                    s1 = fmaf(row[k + 1], v[k + 1], s1);
                }
            } else {
                for (int k = 0; k < bw; k++) s0 = fmaf(row[k], v[k], s0);
            }
            V[(size_t)q * n + i] -= s0 + s1;
        }
    };
    __syncthreads();
    // forward: y_k = (v_k - sum_{j<k} L'_kj y_j) / L'_kk
    if (warp < r) fetch(0, min(32, n));
    for (int b0 = 0; b0 < n; b0 += 32) {
        const int bw = min(32, n - b0);
        if (warp < r) {
            float d = 1.f;
#pragma unroll
            for (int k = 0; k < 32; k++)
                if (lane == k && k < bw) d = f[k];
            const float inv = 1.f / d;
            // a subnormal pivot below 2^-128 has no FP32 reciprocal: such a block divides
            const bool divide = __any_sync(0xffffffffu, isinf(inv));
            for (int q = warp; q < r; q += nw) {
                float v = lane < bw ? V[(size_t)q * n + b0 + lane] : 0.f;
                if (!divide) {
#pragma unroll
                    for (int k = 0; k < 32; k++) {
                        const float y = v * inv, yk = __shfl_sync(0xffffffffu, y, k);
                        v = lane == k ? y : (lane > k ? fmaf(-f[k], yk, v) : v);
                    }
                } else {
                    for (int k = 0; k < bw; k++) {
                        const float yk = __shfl_sync(0xffffffffu, v, k) / __shfl_sync(0xffffffffu, d, k);
                        if (lane == k) v = yk;
                        if (lane > k && lane < bw) v = fmaf(-F[(size_t)(b0 + lane) * fs + b0 + k], yk, v);
                    }
                }
                if (lane < bw) V[(size_t)q * n + b0 + lane] = v;
            }
            if (b0 + 32 < n) fetch(b0 + 32, min(32, n - b0 - 32));
        }
        __syncthreads();
        update(b0 + bw, n, b0, bw);
        __syncthreads();
    }
    // backward: x_k = y_k - sum_{j>k} U'_kj x_j
    if (warp < r) fetch(max(0, n - 32), min(32, n));
    for (int be = n; be > 0; be -= 32) {
        const int b0 = max(0, be - 32), bw = be - b0;
        if (warp < r) {
            for (int q = warp; q < r; q += nw) {
                float v = lane < bw ? V[(size_t)q * n + b0 + lane] : 0.f;
#pragma unroll
                for (int k = 31; k >= 0; k--) {
                    const float xk = __shfl_sync(0xffffffffu, v, k);
                    if (lane < k && k < bw) v = fmaf(-f[k], xk, v);
                }
                if (lane < bw) V[(size_t)q * n + b0 + lane] = v;
            }
            if (b0 > 0) fetch(max(0, b0 - 32), min(32, b0));
        }
        __syncthreads();
        update(0, b0, b0, bw);
        __syncthreads();
    }
}

// R = B - A X (FP64, warp per row; R and X r vectors of n) and the HPL norms:
// per right-hand side max|r|, max|x|; with `first`, also max|b| and ||A||_inf
__device__ void ir_residual(const double *A, long ld, int n, int r, const double *X, double *R, bool first,
                            double *s_red, double *rmax, double *xmax, double *bmax, double *anorm)
{
    const int T = blockDim.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = T >> 5;
    const int stride = 2 * IR_MAX_RHS + 1;  // s_red: per warp the maxima of |r|, of |b|, and of the row sums
    if (lane < stride) s_red[warp * stride + lane] = 0.0;
    __syncwarp();
    for (int i = warp; i < n; i += nw) {
        const double *row = A + (size_t)i * ld;
        for (int q = 0; q < r; q++) {
            const double *x = X + (size_t)q * n;
            double s0 = 0.0, s1 = 0.0, sa = 0.0;
            int j = lane;
            for (; j + 32 < n; j += 64) {
                const double a0 = row[j], a1 = row[j + 32];
                s0 = fma(a0, x[j], s0);
                s1 = fma(a1, x[j + 32], s1);
                sa += fabs(a0) + fabs(a1);
            }
            if (j < n) {
                s0 = fma(row[j], x[j], s0);
                sa += fabs(row[j]);
            }
            s0 += s1;
            for (int o = 16; o > 0; o >>= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
            if (first && q == 0) {
                for (int o = 16; o > 0; o >>= 1) sa += __shfl_xor_sync(0xffffffffu, sa, o);
                if (lane == 0) s_red[warp * stride + 2 * IR_MAX_RHS] = fmax(s_red[warp * stride + 2 * IR_MAX_RHS], sa);
            }
            if (lane == 0) {
                const double b = row[n + q], res = b - s0;
                R[(size_t)q * n + i] = res;
                s_red[warp * stride + q] = fmax(s_red[warp * stride + q], fabs(res));
                s_red[warp * stride + IR_MAX_RHS + q] = fmax(s_red[warp * stride + IR_MAX_RHS + q], fabs(b));
            }
        }
    }
    for (int q = warp; q < r; q += nw) {
        double xm = 0.0;
        for (int i = lane; i < n; i += 32) xm = fmax(xm, fabs(X[(size_t)q * n + i]));
        for (int o = 16; o > 0; o >>= 1) xm = fmax(xm, __shfl_xor_sync(0xffffffffu, xm, o));
        if (lane == 0) xmax[q] = xm;
    }
    __syncthreads();
    if (tid < r) {
        double m1 = 0.0, m2 = 0.0, m3 = 0.0;
        for (int w = 0; w < nw; w++) {
            m1 = fmax(m1, s_red[w * stride + tid]);
            m2 = fmax(m2, s_red[w * stride + IR_MAX_RHS + tid]);
            m3 = fmax(m3, s_red[w * stride + 2 * IR_MAX_RHS]);
        }
        rmax[tid] = m1;
        if (first) {
            bmax[tid] = m2;
            if (tid == 0) *anorm = m3;
        }
    }
    __syncthreads();
}

// (512 threads is the largest launch shape; 128 registers, so one CTA of 512 or
// two of 256 on an SM: held to 64 registers it spills 800 bytes)
__global__ void __launch_bounds__(512)
batch_ir_kernel(double *data, const BatchSys *sys, const long long *woff, uint8_t *arena, const int *order, int count,
                int *counter, int *info, int *iters, int pw, long smem_floats, int max_iter)
{
    extern __shared__ __align__(16) float ism[];
    __shared__ float s_v[4];
    __shared__ int s_i[4];
    __shared__ int s_next, s_zero, s_done;
    __shared__ float s_dinv[64];
    __shared__ BatchPlan s_plan;
    __shared__ double s_red[32 * (2 * IR_MAX_RHS + 1)];
    __shared__ double s_rmax[IR_MAX_RHS], s_xmax[IR_MAX_RHS], s_bmax[IR_MAX_RHS], s_anorm;
    const int T = blockDim.x, tid = threadIdx.x;
    for (;;) {
        if (tid == 0) s_next = atomicAdd(counter, 1);
        __syncthreads();
        const int qi = s_next;
        __syncthreads();
        if (qi >= count) break;
        const int si = order[qi];
        const BatchSys S = sys[si];
        const int n = S.n, r = S.nrhs;
        double *A = data + S.off;
        uint8_t *w = arena + woff[si];
        float *Fg = reinterpret_cast<float *>(w);
        int *perm = reinterpret_cast<int *>(w + ir_align16((size_t)n * n * 4));  // original row of each final row
        double *X = reinterpret_cast<double *>(w + ir_align16((size_t)n * n * 4) + ir_align16((size_t)n * 4));
        double *R = X + (size_t)n * r;
        // in shared memory with an odd row stride (a column's rows in distinct banks)
        const int fso = n | 1;
        const bool in_smem = (long)n * fso + (long)n * r <= smem_floats;
        const int fs = in_smem ? fso : n;
        float *F = in_smem ? ism : Fg;
        float *V = in_smem ? ism + (size_t)n * fs : ism + (size_t)pw * 64 + (size_t)n * (pw + 1);
        if (tid == 0) s_zero = 0;
        for (int i = tid >> 5; i < n; i += T >> 5)
            for (int j = tid & 31; j < n; j += 32) F[(size_t)i * fs + j] = (float)A[(size_t)i * S.ld + j];
        int *order_s = reinterpret_cast<int *>(V);  // perm while it is made (V is not in use yet)
        for (int i = tid; i < n; i += T) order_s[i] = i;
        __syncthreads();
        if (in_smem)
            ir_factor_smem(F, n, fs, order_s, &s_zero);
        else
            ir_factor_blocked(F, n, pw, ism + (size_t)pw * 64, ism, order_s, s_dinv, &s_zero, s_v, s_i, s_plan);
        __syncthreads();
        for (int i = tid; i < n; i += T) perm[i] = order_s[i];
        int it = 0;
        if (s_zero == 0) {
            // x_0 = 0, r_0 = b (the residual of zero also gives the norms of A and b)
            for (int idx = tid; idx < n * r; idx += T) X[idx] = 0.0;
            __syncthreads();
            ir_residual(A, S.ld, n, r, X, R, true, s_red, s_rmax, s_xmax, s_bmax, &s_anorm);
            for (it = 1; it <= max_iter; it++) {
                for (int i = tid; i < n; i += T) {
                    const int from = perm[i];
                    for (int q = 0; q < r; q++) V[(size_t)q * n + i] = (float)R[(size_t)q * n + from];
                }
                ir_solve(F, n, fs, V, r);
                for (int idx = tid; idx < n * r; idx += T) X[idx] += (double)V[idx];
                __syncthreads();
                ir_residual(A, S.ld, n, r, X, R, false, s_red, s_rmax, s_xmax, s_bmax, &s_anorm);
                if (tid == 0) {
                    bool ok = true;
                    // lu2's bar of 16 with room for the rounding of a residual: summed with k
                    // roundings it is off by at most k u (|A||x| + |b|), k / n in units of h; k
                    // is at most n / 64 + 9 here and n + 1 wherever the caller sums it (held
                    // to 16 itself, 1 of 20,000 systems came back at 16.01)
                    const double bar = 16 * n - (n + 1 + min(n + 1, n / 64 + 9));  // of n h
                    for (int q = 0; q < r; q++) {
                        const double h = s_rmax[q] / (1.1102230246251565e-16 * (s_anorm * s_xmax[q] + s_bmax[q]));
                        if (!(h < bar)) ok = false;
                    }
                    s_done = ok;
                }
                __syncthreads();
                if (s_done) break;
            }
            if (it > max_iter) it = max_iter;
            for (int idx = tid; idx < n * r; idx += T) {
                const int q = idx / n, i = idx - q * n;
                A[(size_t)i * S.ld + n + q] = X[idx];
            }
        }
        if (tid == 0) {
            info[si] = s_zero;
            iters[si] = it;
        }
        __syncthreads();
    }
}

long batch_ir_smem_floats(const BatchSys *sys, int count, int pw, long floor_floats)
{
    long need = floor_floats;
    for (int i = 0; i < count; i++) {
        const long b = (long)pw * 64 + (long)sys[i].n * (pw + 1) + (long)sys[i].n * sys[i].nrhs;
        if (b > need) need = b;
    }
    return need;
}

cudaError_t batch_ir_grid(int threads, long smem_floats, int ctas_per_sm, int count, int *grid)
{
    if (threads < 64 || threads > 512 || (threads & 31)) return cudaErrorInvalidValue;
    const size_t smem = (size_t)smem_floats * sizeof(float);
    if (smem > BATCH_SMEM_MAX) return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(batch_ir_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, BATCH_SMEM_MAX);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 148;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    int occ = 0;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, batch_ir_kernel, threads, smem)) != cudaSuccess)
        return e;
    if (occ < 1) return cudaErrorInvalidConfiguration;
    if (ctas_per_sm > occ || ctas_per_sm < 1) ctas_per_sm = occ;
    const int g = sms * ctas_per_sm;
    *grid = g > count ? count : g;
    return cudaSuccess;
}

cudaError_t launch_batch_ir(double *data, const BatchSys *sys, const long long *woff, uint8_t *arena,
                            const int *order, int count, int *counter, int *info, int *iters, long smem_floats, int pw,
                            int threads, int grid, int max_iter, cudaStream_t st)
{
    if (count <= 0) return cudaSuccess;
    if (pw < 16 || pw > 64 || threads < 64 || threads > 512 || (threads & 31) || grid < 1 || max_iter < 1 ||
        (size_t)smem_floats * sizeof(float) > BATCH_SMEM_MAX)
        return cudaErrorInvalidValue;
    cudaError_t e = cudaMemsetAsync(counter, 0, sizeof(int), st);
    if (e != cudaSuccess) return e;
    count_launch();
    batch_ir_kernel<<<grid, threads, (size_t)smem_floats * sizeof(float), st>>>(
        data, sys, woff, arena, order, count, counter, info, iters, pw, smem_floats, max_iter);
    return cudaGetLastError();
}

}  // namespace lu2gpu

// kernels_trisolve.cu -- triangular solves with stored factors, one persistent
// cooperative launch each.
//
//   upper: x = U'^{-1} y with the unit upper factor, lu2's backward_sub
//          (lu2.c:110-116)
//   lower: the forward solve lu2 applies to its augmented columns (per panel
//          the pivots with the 1/pivot scaling, the unit-lower solve and the
//          update of the rows below, lu2.c:524-581) on stored factors
//
// Rows are cut into blocks of at most 128 (the lower solve: inside its
// panels), numbered in the order they are solved; block p belongs to CTA p mod
// G of a cooperative grid of G co-resident CTAs, which keeps the right-hand
// sides of all its blocks in shared memory.  The blocks' solutions x_p are
// published in the order p = 0, 1, 2, ...: when x_p is out, every CTA
// subtracts M(block q, block p) x_p from each of its blocks q > p, in that
// order, so every element receives its updates in a fixed order; the CTA owning
// block p+1 does that block first and solves it at once.  Each tile of M is
// read once: a CTA loads the tile its next block takes from a source before it
// waits for that source's x (the tiles do not depend on x).
// Publication: the solving warps store the block's x straight from their
// registers into its slots as stamped words (the call's epoch beside each
// 32-bit half, no fence); a reader re-loads them until all carry the epoch
// (bounded wait), which gives it x in the same round trip.
//
// What bounds it: the chain of blocks, one solve, one publication and one
// tile product each -- not the factor's bytes.  Hence
//  * 128 rows a block: the publication, about 1 us through L2, is paid half as
//    often as with 64;
//  * a block's solve runs in four warps per right-hand side, 32 rows each: a
//    warp finishes its triangle four columns at a time (their values shuffled
//    to all lanes together and finished there redundantly, so that a column
//    costs a quarter of a shuffle's latency), then the later warps subtract its
//    32 columns.  One warp walking all 128 rows took 11800 cycles a block;
//  * FP64 tile products run on the tensor pipe (mma.sync m16n8k8, always eight
//    right-hand sides wide, so that a column's result does not depend on how
//    many there are): read from shared memory by every thread, x cost 8600
//    cycles a block with 4 right-hand sides; the tensor pipe takes 2050 with
//    any number, the CUDA cores 1250 with one.
//
// The FP64 lower solve repeats the factorization's own operations on a riding
// column in the same order, so that a re-solve gives what the factorization
// gave (with the shipped reference's pivots anything else differs visibly):
// inside a panel the 16-row blocks of trsm_dmma_kernel (16 products summed
// from zero, then subtracted), across panels the trailing update's own MMA
// with its permuted k, accumulating on the right-hand side column after column.
//
// The lower solve's rows.  Earlier panels' L columns are not swapped by later
// panels (lu2.c:543-553): the row that ends at position f sat at position
// row(P, f) right after panel P.  Right-hand sides are kept in final
// positions and a tile's rows are gathered through that map (512-byte
// segments or more), so no exchange is left in the chain.  launch_solve_plan
// builds the map for all panels at once from the pivots.
#include "lu2gpu_internal.cuh"

namespace lu2gpu {

constexpr int TS_B = 128;         // rows per block
constexpr int TS_THREADS = 512;
constexpr int TS_TLD = TS_B + 1;  // pitch of the diagonal block in shared memory
constexpr int TS_E = TS_B / 4;    // elements of a tile per thread
constexpr int TS_XQ = TS_B + 8;   // pitch of a source's x per right-hand side: B fragments on distinct banks

template <typename T>
struct TriParams {
    const T *a;
    long ld;
    int n, nb, bpp, nblk;  // panel width, blocks per panel
    const T *y;            // right-hand sides (row stride ldy), columns of this launch
    long ldy;
    T *x;
    long ldx;
    int nr;
    const int *rows;  // lower: positions before each panel, by final position (solve_map_at)
    const T *dinv;    // lower: 1/pivot
    unsigned long long *xslots;  // element (row, q) at 2 (row BS_MAXR + q)
    unsigned epoch;
    int *status;
};

// two consecutive elements
__device__ __forceinline__ void ts_ld2(const double *p, double &a, double &b)
{
    const double2 w = __ldg(reinterpret_cast<const double2 *>(p));
    a = w.x;
    b = w.y;
}
__device__ __forceinline__ void ts_ld2(const float *p, float &a, float &b)
{
    const float2 w = __ldg(reinterpret_cast<const float2 *>(p));
    a = w.x;
    b = w.y;
}

__device__ __forceinline__ unsigned ts_smem32(const void *p)
{
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void ts_lds(unsigned p, double &v) { asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(p)); }
__device__ __forceinline__ void ts_lds(unsigned p, float &v) { asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(p)); }
__device__ __forceinline__ void ts_lds2(unsigned p, double &a, double &b)
{
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(a), "=d"(b) : "r"(p));
}
__device__ __forceinline__ void ts_lds2(unsigned p, float &a, float &b)
{
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(a), "=f"(b) : "r"(p));
}

__device__ __forceinline__ void ts_mma(double (&c)[4], double a0, double a1, double a2, double a3, double b0, double b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a0), "d"(a1), "d"(a2), "d"(a3), "d"(b0), "d"(b1));
}

// NR = 1 (FP32): one right-hand side on the CUDA cores; NR = 8 (FP64): up to 8,
// padded with zeros, on the tensor pipe.  EXACT: the FP64 lower solve.
template <typename T, bool LOWER, int NR>
__global__ void __launch_bounds__(TS_THREADS, 1) tri_solve_kernel(const TriParams<T> P)
{
    constexpr bool MMA = NR == 8, EXACT = LOWER && sizeof(T) == 8;
    static_assert(!EXACT || MMA, "the factorization's order of operations is the MMA's");
    static_assert(!MMA || sizeof(T) == 8, "FP64 MMA");
    extern __shared__ __align__(16) unsigned char ts_smem[];
    const int G = gridDim.x, cta = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nblk = P.nblk;
    const int n_own = cta < nblk ? (nblk - cta + G - 1) / G : 0;
    constexpr int XB = TS_XQ * NR;
    T *Td = reinterpret_cast<T *>(ts_smem);      // [TS_B][TS_TLD], the owned diagonal block solved next
    T *xs = Td + TS_B * TS_TLD;                  // [2][NR][TS_XQ]
    T *part_sum = xs + 2 * XB;                   // [TS_B][NR] (tensor pipe, not EXACT)
    T *acc = part_sum + (MMA && !EXACT ? TS_B * NR : 0);  // [n_own][TS_B][NR]
    T *sdinv = acc + (size_t)n_own * TS_B * NR;  // [n_own][TS_B] (lower)
    // an earlier wait or check of this call failed: nothing to do
    if (__syncthreads_or(tid == 0 && *(volatile int *)&P.status[1] != 0)) return;

    // block p in solve order: its panel, first row, rows
    auto panel_of = [&](int p) { return LOWER ? p / P.bpp : 0; };
    auto r0_of = [&](int p) {
        if constexpr (LOWER) return p / P.bpp * P.nb + p % P.bpp * TS_B;
        return (nblk - 1 - p) * TS_B;
    };
    auto rows_of = [&](int p) {
        const int r0 = r0_of(p);
        int rows = min(TS_B, P.n - r0);
        if (LOWER) rows = min(rows, P.nb - p % P.bpp * TS_B);
        return rows;
    };

    for (int k = 0; k < n_own; k++) {
        const int p = cta + k * G, r0 = r0_of(p), rows = rows_of(p);
        for (int e = tid; e < TS_B * NR; e += TS_THREADS) {
            const int r = e / NR, q = e % NR;
            T v = T(0);
            if (r < rows && q < P.nr) {
                const int from = LOWER ? __ldg(P.rows + r0 + r) : r0 + r;  // the row's original position
                v = P.y[(size_t)from * P.ldy + q];
            }
            acc[((size_t)k * TS_B + r) * NR + q] = v;
        }
        if (LOWER)
            for (int r = tid; r < TS_B; r += TS_THREADS)
                sdinv[k * TS_B + r] = r < rows ? P.dinv[r0 + r] : T(1);
    }
    for (int e = tid; e < 2 * XB; e += TS_THREADS) xs[e] = T(0);  // right-hand sides past nr stay zero

    // owned block k's diagonal block into Td (issued right after the previous
    // solve, off the critical path), zero outside its strict triangle
    auto prefetch_diag = [&](int k) {
        const int p = cta + k * G, r0 = r0_of(p), rows = rows_of(p);
        for (int e = tid; e < TS_B * TS_B; e += TS_THREADS) {
            const int r = e / TS_B, c = e % TS_B;
            T *d = &Td[r * TS_TLD + c];
            if (r < rows && c < rows && (LOWER ? c < r : c > r)) {
                const unsigned dst = (unsigned)__cvta_generic_to_shared(d);
                if constexpr (sizeof(T) == 8)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst),
                                 "l"(P.a + (size_t)(r0 + r) * P.ld + r0 + c)
                                 : "memory");
                else
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst),
                                 "l"(P.a + (size_t)(r0 + r) * P.ld + r0 + c)
                                 : "memory");
            } else {
                *d = T(0);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    // solve owned block k (all updates applied) into xs[buf] and x: four warps
    // per right-hand side q (then q + 4), warp m of them with rows 32 m ..
    // 32 m + 31, one per lane.  (m is rotated with q: the warps whose turn it
    // is at the same time sit on different schedulers.)
    auto solve = [&](int k, int buf) {
        const int p = cta + k * G, r0 = r0_of(p), rows = rows_of(p);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        const int m = (warp + (warp >> 2)) & 3, r = 32 * m + lane;
        const unsigned td = ts_smem32(Td), tr = td + r * TS_TLD * (unsigned)sizeof(T);
        unsigned long long *slot = P.xslots + (size_t)r0 * (2 * BS_MAXR);
#pragma unroll 1
        for (int q = warp >> 2; q < NR && q < P.nr; q += 4) {
            T *X = xs + buf * XB + q * TS_XQ;
            const unsigned xq = ts_smem32(X);
            T y = acc[((size_t)k * TS_B + r) * NR + q];
            if (LOWER && p % P.bpp == 0) y *= sdinv[k * TS_B + r];  // a panel's first block: nothing scaled it yet
#pragma unroll 1
            for (int jj = 0; jj < 4; jj++) {
                const int j = LOWER ? jj : 3 - jj;  // the warp whose turn it is
                if (32 * j >= rows) continue;
                if (m == j) {
                    T s = T(0);  // EXACT: the first 16 columns' products for the later 16 rows
                    // group ll's columns in solve order, the lane's row and the 4 x 4 triangle,
                    // read one group ahead
                    T tc[4], tt[6];
                    auto fetch = [&](int ll) {
                        const int c0 = 32 * j + (LOWER ? ll : 28 - ll);
#pragma unroll
                        for (int e = 0; e < 4; e++) ts_lds(tr + (c0 + (LOWER ? e : 3 - e)) * (unsigned)sizeof(T), tc[e]);
#pragma unroll
                        for (int e = 1; e < 4; e++)
#pragma unroll
                            for (int f = 0; f < e; f++) {
                                const int re = c0 + (LOWER ? e : 3 - e), cf = c0 + (LOWER ? f : 3 - f);
                                ts_lds(td + (re * TS_TLD + cf) * (unsigned)sizeof(T), tt[e * (e - 1) / 2 + f]);
                            }
                    };
                    fetch(0);
#pragma unroll
                    for (int ll = 0; ll < 32; ll += 4) {
                        const int l0 = LOWER ? ll : 28 - ll;
                        T xv[4], cc[4], ct[6];
#pragma unroll
                        for (int e = 0; e < 4; e++) xv[e] = __shfl_sync(0xffffffffu, y, l0 + (LOWER ? e : 3 - e));
#pragma unroll
                        for (int e = 0; e < 4; e++) cc[e] = tc[e];
#pragma unroll
                        for (int e = 0; e < 6; e++) ct[e] = tt[e];
                        if (ll + 4 < 32) fetch(ll + 4);
#pragma unroll
                        for (int e = 1; e < 4; e++)
#pragma unroll
                            for (int f = 0; f < e; f++) xv[e] = fma(-ct[e * (e - 1) / 2 + f], xv[f], xv[e]);
                        const bool far = EXACT && ll < 16 && lane >= 16;
                        T v = far ? s : y;
#pragma unroll
                        for (int e = 0; e < 4; e++) v = fma(far ? cc[e] : -cc[e], xv[e], v);
                        s = far ? v : s;
                        const T yf = y - s;
                        y = far ? (ll == 12 ? yf : y) : ((LOWER ? lane > l0 + 3 : lane < l0) ? v : y);
#pragma unroll
                        for (int e = 0; e < 4; e++) y = lane == l0 + (LOWER ? e : 3 - e) ? xv[e] : y;
                    }
                    X[r] = r < rows ? y : T(0);
                }
                asm volatile("bar.sync %0, 128;" ::"r"(1 + (warp >> 2)) : "memory");
                if (LOWER ? m > j : m < j) {
                    // two chains of 16 products
                    const unsigned tj = tr + 32 * j * (unsigned)sizeof(T), xj = xq + 32 * j * (unsigned)sizeof(T);
                    T s0 = T(0), s1 = T(0);
#pragma unroll
                    for (int e = 0; e < 16; e += 2) {
                        T x0, x1, x2, x3, t0, t1, t2, t3;
                        ts_lds2(xj + e * (unsigned)sizeof(T), x0, x1);
                        ts_lds2(xj + (16 + e) * (unsigned)sizeof(T), x2, x3);
                        ts_lds(tj + e * (unsigned)sizeof(T), t0);
                        ts_lds(tj + (e + 1) * (unsigned)sizeof(T), t1);
                        ts_lds(tj + (16 + e) * (unsigned)sizeof(T), t2);
                        ts_lds(tj + (17 + e) * (unsigned)sizeof(T), t3);
                        s0 = fma(t0, x0, s0);
                        s1 = fma(t2, x2, s1);
                        s0 = fma(t1, x1, s0);
                        s1 = fma(t3, x3, s1);
                    }
                    y -= s0;
                    y -= s1;
                }
                if (m == j && r < rows) {  // published beside the next warp's work
                    st_stamped(slot + 2 * (r * BS_MAXR + q), P.epoch, (double)y);
                    P.x[(size_t)(r0 + r) * P.ldx + q] = y;
                }
            }
        }
        __syncthreads();
        if (k + 1 < n_own) prefetch_diag(k + 1);
    };

    // The thread's part of a tile.  CUDA cores: row tid / 4, column pairs
    // 8 j + 2 (tid % 4), of which the four threads of a row read 64 (float: 32)
    // contiguous bytes per load.  Tensor pipe: the A fragments of rows
    // 16 (warp % 8) + g, + 8 and columns 64 (warp / 8) + 8 j + {2 t, 2 t + 1}
    // (the trailing update's permuted k), or, EXACT inside a panel, {t, t + 4}.
    const int g = lane >> 2, t = lane & 3;
    const int tr0 = MMA ? 16 * (warp & 7) + g : tid >> 2, half = warp >> 3;
    constexpr int NROW = MMA ? 2 : 1;  // rows tr0, tr0 + 8
    auto tile_rows = [&](int k, int p_src, int (&row)[NROW]) {
        const int p = cta + k * G;
#pragma unroll
        for (int h = 0; h < NROW; h++) {
            const int r = r0_of(p) + tr0 + 8 * h;
            if (tr0 + 8 * h >= rows_of(p))
                row[h] = -1;
            else if (!LOWER || panel_of(p) == panel_of(p_src))
                row[h] = r;
            else
                row[h] = __ldg(P.rows + solve_map_at(panel_of(p_src) + 1, P.n, P.nb) + r);  // after the source's panel
        }
    };
    const bool vec = ((reinterpret_cast<uintptr_t>(P.a) & (2 * sizeof(T) - 1)) == 0) && ((P.ld & 1) == 0) &&
                     (!LOWER || (P.nb & 1) == 0);
    auto load_tile = [&](int k, const int (&row)[NROW], int p_src, T (&v)[TS_E]) {
        const int c0 = r0_of(p_src), cols = rows_of(p_src);
        const bool natural = EXACT && panel_of(cta + k * G) == panel_of(p_src);
#pragma unroll
        for (int h = 0; h < NROW; h++) {
            const int first = MMA ? 64 * half + (natural ? t : 2 * t) : 2 * (tid & 3);
            const int second = natural ? 4 : 1;
            const T *u = P.a + (size_t)max(row[h], 0) * P.ld + c0 + first;
#pragma unroll
            for (int j = 0; j < TS_E / 2 / NROW; j++) {
                T &v0 = v[2 * (j * NROW + h)], &v1 = v[2 * (j * NROW + h) + 1];
                v0 = v1 = T(0);
                if (row[h] >= 0) {
                    if (vec && !natural && cols == TS_B) {
                        ts_ld2(u + 8 * j, v0, v1);
                    } else {
                        const int col = first + 8 * j;
                        if (col < cols) v0 = __ldg(u + 8 * j);
                        if (col + second < cols) v1 = __ldg(u + 8 * j + second);
                    }
                }
            }
        }
    };
    // acc[k] -= tile * X; the first source of the block's own panel finds it
    // updated by all earlier panels and scales it by 1/pivot before
    auto apply_tile = [&](int k, int p_src, const T (&v)[TS_E], const T *X) {
        const int p = cta + k * G;
        const bool own = LOWER && panel_of(p_src) == panel_of(p);
        const bool scale = own && p_src % P.bpp == 0;
        T *A = acc + (size_t)k * TS_B * NR;
        if constexpr (MMA) {
            double c[4];
            double *o0 = A + tr0 * NR + 2 * t, *o1 = o0 + 8 * NR;  // rows tr0, tr0 + 8, right-hand sides 2t, 2t + 1
            const double *xg = X + g * TS_XQ + 64 * half;           // B: k by 8 j + ..., column g
            auto get = [&]() {
                c[0] = o0[0];
                c[1] = o0[1];
                c[2] = o1[0];
                c[3] = o1[1];
            };
            auto put = [&]() {
                o0[0] = c[0];
                o0[1] = c[1];
                o1[0] = c[2];
                o1[1] = c[3];
            };
            auto products = [&]() {  // c -= tile half * X
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const double2 x = *reinterpret_cast<const double2 *>(xg + 8 * j + 2 * t);
                    ts_mma(c, v[4 * j], v[4 * j + 2], v[4 * j + 1], v[4 * j + 3], -x.x, -x.y);
                }
            };
            if constexpr (!EXACT) {
                // four chains of 16 products: one chain of 64 left a backward
                // error of x up to half larger (n = 2048, 16 systems, geometric
                // mean: 6.1e-16 against 4.6e-16)
                double s[4][4];
#pragma unroll
                for (int b = 0; b < 4; b++) s[b][0] = s[b][1] = s[b][2] = s[b][3] = 0.0;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const double2 x = *reinterpret_cast<const double2 *>(xg + 8 * j + 2 * t);
                    ts_mma(s[j & 3], v[4 * j], v[4 * j + 2], v[4 * j + 1], v[4 * j + 3], -x.x, -x.y);
                }
#pragma unroll
                for (int e = 0; e < 4; e++) c[e] = (s[0][e] + s[1][e]) + (s[2][e] + s[3][e]);
                double *q0 = part_sum + tr0 * NR + 2 * t, *q1 = q0 + 8 * NR;
                if (half == 1) {
                    q0[0] = c[0];
                    q0[1] = c[1];
                    q1[0] = c[2];
                    q1[1] = c[3];
                }
                __syncthreads();
                if (half == 0) {
                    o0[0] += c[0] + q0[0];
                    o0[1] += c[1] + q0[1];
                    o1[0] += c[2] + q1[0];
                    o1[1] += c[3] + q1[1];
                }
                __syncthreads();  // part_sum is free again
            } else if (!own) {
                if (half == 0) {
                    get();
                    products();
                    put();
                }
                __syncthreads();
                if (half == 1) {
                    get();
                    products();
                    put();
                }
            } else {
                double s[4][4];  // 16 columns each
#pragma unroll
                for (int b = 0; b < 4; b++) {
                    s[b][0] = s[b][1] = s[b][2] = s[b][3] = 0.0;
#pragma unroll
                    for (int j = 2 * b; j < 2 * b + 2; j++)
                        ts_mma(s[b], v[4 * j], v[4 * j + 2], v[4 * j + 1], v[4 * j + 3], xg[8 * j + t],
                               xg[8 * j + t + 4]);
                }
                if (half == 0) {
                    get();
                    if (scale) {
                        const double d0 = sdinv[k * TS_B + tr0], d1 = sdinv[k * TS_B + tr0 + 8];
                        c[0] *= d0;
                        c[1] *= d0;
                        c[2] *= d1;
                        c[3] *= d1;
                    }
#pragma unroll
                    for (int b = 0; b < 4; b++)
#pragma unroll
                        for (int e = 0; e < 4; e++) c[e] -= s[b][e];
                    put();
                }
                __syncthreads();
                if (half == 1) {
                    get();
#pragma unroll
                    for (int b = 0; b < 4; b++)
#pragma unroll
                        for (int e = 0; e < 4; e++) c[e] -= s[b][e];
                    put();
                }
            }
        } else {
            T s[NR];
#pragma unroll
            for (int q = 0; q < NR; q++) {
                const T *xq = X + q * TS_XQ + 2 * (tid & 3);
                T s0 = T(0), s1 = T(0);
#pragma unroll
                for (int j = 0; j < TS_E / 2; j++) {
                    s0 = fma(v[2 * j], xq[8 * j], s0);
                    s1 = fma(v[2 * j + 1], xq[8 * j + 1], s1);
                }
                s[q] = s0 + s1;
                s[q] += __shfl_xor_sync(0xffffffffu, s[q], 1);
                s[q] += __shfl_xor_sync(0xffffffffu, s[q], 2);
            }
            if ((tid & 3) == 0 && tr0 < rows_of(p)) {
                const T d = scale ? sdinv[k * TS_B + tr0] : T(1);
#pragma unroll
                for (int q = 0; q < NR; q++) {
                    T &o = A[tr0 * NR + q];
                    o = (scale ? o * d : o) - s[q];
                }
            }
        }
    };

    int next = 0;
    if (n_own > 0) prefetch_diag(0);
    __syncthreads();
    if (n_own > 0 && cta == 0) {  // the first block needs no update
        solve(0, 0);
        next = 1;
    }
    const unsigned long long t0 = globaltimer_ns();
    int row[NROW];
#pragma unroll
    for (int h = 0; h < NROW; h++) row[h] = -1;
    if (next < n_own) tile_rows(next, 0, row);
    for (int p_src = 0; p_src < nblk; p_src++) {
        const int buf = p_src & 1;
        T *X = xs + buf * XB;
        const int k_first = next;
        T v[TS_E];
        if (k_first < n_own) {
            load_tile(k_first, row, p_src, v);
            if (p_src + 1 < nblk) tile_rows(k_first, p_src + 1, row);
        }
        if (p_src % G != cta && k_first < n_own) {
            // the source block's x from its slots: each thread re-loads its
            // elements until they carry this call's epoch; the CTA agrees on
            // completion, or on giving up, at one barrier per round
            const unsigned long long *slot = P.xslots + (size_t)r0_of(p_src) * (2 * BS_MAXR);
            const int rows = rows_of(p_src);
            constexpr int EPT = (TS_B * NR + TS_THREADS - 1) / TS_THREADS;  // elements per thread
            unsigned todo = 0;
#pragma unroll
            for (int u = 0; u < EPT; u++) {
                const int e = tid + u * TS_THREADS, r = e / NR, q = e % NR;
                if (e >= TS_B * NR || q >= P.nr) continue;
                if (r < rows)
                    todo |= 1u << u;
                else
                    X[q * TS_XQ + r] = T(0);
            }
            for (unsigned round = 1;; round++) {
#pragma unroll
                for (int u = 0; u < EPT; u++) {
                    if (!((todo >> u) & 1u)) continue;
                    const int e = tid + u * TS_THREADS, r = e / NR, q = e % NR;
                    unsigned long long hi, lo;
                    ld_pair(slot + 2 * (r * BS_MAXR + q), hi, lo);
                    if (stamped(hi, P.epoch) && stamped(lo, P.epoch)) {
                        X[q * TS_XQ + r] = (T)unstamp(hi, lo);
                        todo &= ~(1u << u);
                    }
                }
                if (__syncthreads_and(todo == 0)) break;
                const bool late = (round & 63u) == 0 && tid == 0 &&
                                  (*(volatile int *)&P.status[1] != 0 || globaltimer_ns() - t0 > WAIT_LIMIT_NS);
                if ((round & 63u) == 0 && __syncthreads_or(late)) {
                    if (tid == 0 && *(volatile int *)&P.status[1] == 0) record_error(P.status, ERR_BARRIER_TIMEOUT, 6);
                    asm volatile("cp.async.wait_all;" ::: "memory");  // the next diagonal block, on its way to Td
                    return;
                }
            }
        }
        if (k_first < n_own) {
            apply_tile(k_first, p_src, v, X);
            if (cta + k_first * G == p_src + 1) {
                __syncthreads();
                solve(k_first, buf ^ 1);
                next = k_first + 1;
                if (next < n_own && p_src + 1 < nblk) tile_rows(next, p_src + 1, row);
            }
        }
        for (int k = k_first + 1; k < n_own; k++) {
            int rk[NROW];
            tile_rows(k, p_src, rk);
            load_tile(k, rk, p_src, v);
            apply_tile(k, p_src, v, X);
        }
        __syncthreads();  // X (this buffer) is overwritten two sources later
    }
}

// CTAs of a solve of nblk blocks, and the shared memory of one
static int ts_grid(int nblk, int sms) { return nblk < sms ? nblk : sms; }
static size_t ts_bytes(int nblk, int sms, bool lower, int nr, size_t tsize)
{
    const int G = ts_grid(nblk, sms), own = (nblk + G - 1) / G;
    return ((size_t)TS_B * TS_TLD + 2 * TS_XQ * nr + (nr == 8 && !lower ? TS_B * nr : 0) +
            (size_t)own * TS_B * (nr + (lower ? 1 : 0))) *
           tsize;
}
constexpr size_t TS_SMEM_MAX = 220 * 1024;

template <typename T, bool LOWER, int NR>
static cudaError_t ts_launch(TriParams<T> P, cudaStream_t st, bool *used)
{
    *used = false;
    int dev = 0, sms = 148;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    const int G = ts_grid(P.nblk, sms);
    const size_t smem = ts_bytes(P.nblk, sms, LOWER, NR, sizeof(T));
    if (smem > TS_SMEM_MAX) return cudaSuccess;  // too many blocks per CTA: the caller's other way
    auto kern = tri_solve_kernel<T, LOWER, NR>;
    if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TS_SMEM_MAX)) != cudaSuccess)
        return e;
    void *args[] = {&P};
    count_launch();
    e = cudaLaunchCooperativeKernel((const void *)kern, dim3(G), dim3(TS_THREADS), args, smem, st);
    if (e == cudaSuccess) *used = true;
    return e;
}

// right-hand sides one launch takes: FP32 solves, of one vector each, stay on
// the CUDA cores
template <typename T>
static constexpr int ts_maxr()
{
    return sizeof(T) == 8 ? BS_MAXR : 1;
}

template <typename T, bool LOWER>
static cudaError_t ts_any(TriParams<T> P, const BsBuffers &bs, cudaStream_t st, bool *used)
{
    *used = false;
    if (P.n > bs.cap_rows) return cudaSuccess;
    P.xslots = bs.xslots;
    P.status = bs.status;
    P.epoch = ++*bs.epoch;
    if (P.epoch == 0) P.epoch = ++*bs.epoch;
    return ts_launch<T, LOWER, ts_maxr<T>()>(P, st, used);
}

template <typename T>
static cudaError_t upper_t(const T *a, long ld, int n, int nrhs, const T *y, long ldy, T *x, long ldx,
                           const BsBuffers &bs, cudaStream_t st, bool *used)
{
    *used = false;
    for (int c0 = 0; c0 < nrhs; c0 += ts_maxr<T>()) {
        TriParams<T> P{};
        P.a = a;
        P.ld = ld;
        P.n = n;
        P.nb = TS_B;
        P.bpp = 1;
        P.nblk = (n + TS_B - 1) / TS_B;
        P.y = y + c0;
        P.ldy = ldy;
        P.x = x + c0;
        P.ldx = ldx;
        P.nr = nrhs - c0 < ts_maxr<T>() ? nrhs - c0 : ts_maxr<T>();
        const cudaError_t e = ts_any<T, false>(P, bs, st, used);
        if (e != cudaSuccess || !*used) return e;  // the first chunk decides: all have the same blocks
    }
    return cudaSuccess;
}

cudaError_t launch_upper_solve(const double *a, long ld, int n, int nrhs, const double *y, long ldy, double *x, long ldx,
                               const BsBuffers &bs, cudaStream_t st, bool *used)
{
    return upper_t(a, ld, n, nrhs, y, ldy, x, ldx, bs, st, used);
}

cudaError_t launch_upper_solve(const float *a, long ld, int n, int nrhs, const float *y, long ldy, float *x, long ldx,
                               const BsBuffers &bs, cudaStream_t st, bool *used)
{
    return upper_t(a, ld, n, nrhs, y, ldy, x, ldx, bs, st, used);
}

// blocks of the lower solve: every panel of nb rows in blocks of its own
static int lower_blocks(int n, int nb)
{
    const int npan = (n + nb - 1) / nb, last = n - (npan - 1) * nb;
    return (npan - 1) * ((nb + TS_B - 1) / TS_B) + (last + TS_B - 1) / TS_B;
}

static int ts_sms()
{
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0;
    return sms;
}

// Right-hand sides (FP64) up to which the two persistent solves beat the panel
// loop.  A pass of 8 walks the chain of blocks again; the loop's panels cost about
// the same for any of these numbers.  us, persistent / panel loop:
//   one panel, n = 16:  1: 56 / 50, 8: 59 / 51;  64:  1: 57 / 55, 8: 64 / 58 (the row map, two launches, is more
//       than one exchange);  96:  1: 60.6 / 61.0, 4: 61.4 / 62.1, 8: 70 / 66;  128:  1: 62 / 66, 4: 65 / 66, 8: 76 / 73
//   one block of several panels, n = 17, panels of 16:  1: 58 / 63, 8: 62 / 66;  96, of 64:  1: 63 / 75, 8: 73 / 79;
//       100, of 16:  16: 152 / 163, 24: 207 / 178
//   panels of 512, n = 4096:  32: 3293 / 3779 (the loop's block solves are slow there)
//   256:  17: 2044 / 1975 (n = 40000: 20.6 / 21.8 ms), 24: 2463 / 2167
//   128:  17: 2034 / 2115, 24: 2452 / 2279;  64:  17: 2361 / 2427, 24: 2814 / 2636
//   48:  16: 2197 / 2408, 17: 2743 / 2596
//   32:  24: 3313 / 3567, 25: 3984 / 3747; n = 37000, 8 blocks per CTA:  9: 34.5 / 28.1 ms
//   16, n = 2048, one block per CTA:  24: 2648 / 2499-2717, 25: 3200 / 2764; n = 6144, 3:  16: 6054 / 6926,
//       17: 8497 / 7489; n = 10240, 5:  8: 6.2 / 10.6, 9: 11.6 / 11.1-12.1 ms
// (a block is never larger than a panel, and one of 16 rows costs a tile of 128)
int tri_solve_few_rhs(int n, int nb)
{
    if (n <= nb && n <= TS_B) return n <= 64 ? 0 : 4;
    if (n <= TS_B) return nb >= 48 ? BS_MAXR : 16;
    if (nb > 256) return 32;
    if (nb >= 48) return nb >= 64 ? 18 : 16;
    const int sms = ts_sms(), own = sms > 0 ? (lower_blocks(n, nb) + sms - 1) / sms : 1;
    return own > 4 ? BS_MAXR : nb == 32 || own <= 2 ? 24 : 16;
}

bool tri_solves_fit(int n, int nb, size_t tsize)
{
    const int sms = ts_sms();
    if (sms <= 0) return false;
    const int nr = tsize == sizeof(double) ? ts_maxr<double>() : ts_maxr<float>();
    return ts_bytes(lower_blocks(n, nb), sms, true, nr, tsize) <= TS_SMEM_MAX &&
           ts_bytes((n + TS_B - 1) / TS_B, sms, false, nr, tsize) <= TS_SMEM_MAX;
}

template <typename T>
static cudaError_t lower_t(const T *a, long ld, int n, int nb, const int *rows, const T *dinv, const T *b, long ldb,
                           int nrhs, T *y, long ldy, const BsBuffers &bs, cudaStream_t st, bool *used)
{
    *used = false;
    if (nrhs > ts_maxr<T>()) return cudaErrorInvalidValue;
    TriParams<T> P{};
    P.a = a;
    P.ld = ld;
    P.n = n;
    P.nb = nb;
    P.bpp = (nb + TS_B - 1) / TS_B;
    P.nblk = lower_blocks(n, nb);
    P.y = b;
    P.ldy = ldb;
    P.x = y;
    P.ldx = ldy;
    P.nr = nrhs;
    P.rows = rows;
    P.dinv = dinv;
    return ts_any<T, true>(P, bs, st, used);
}

cudaError_t launch_lower_solve(const double *a, long ld, int n, int nb, const int *rows, const double *dinv,
                               const double *b, long ldb, int nrhs, double *y, long ldy, const BsBuffers &bs,
                               cudaStream_t st, bool *used)
{
    return lower_t(a, ld, n, nb, rows, dinv, b, ldb, nrhs, y, ldy, bs, st, used);
}

cudaError_t launch_lower_solve(const float *a, long ld, int n, int nb, const int *rows, const float *dinv,
                               const float *b, long ldb, int nrhs, float *y, long ldy, const BsBuffers &bs,
                               cudaStream_t st, bool *used)
{
    return lower_t(a, ld, n, nb, rows, dinv, b, ldb, nrhs, y, ldy, bs, st, used);
}

}  // namespace lu2gpu

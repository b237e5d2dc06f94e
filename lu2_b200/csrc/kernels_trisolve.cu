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
// tile product each -- not the factor's bytes.  Hence 128 rows a block (the
// publication, about 1.5 us through L2, is paid half as often as with 64), and
// the diagonal block solved four columns at a time: their four values are
// shuffled to all lanes together and finished there redundantly, so a column
// costs a quarter of a shuffle's latency.
//
// The FP64 lower solve repeats the factorization's own operations on a riding
// column in the same order, so that a re-solve gives what the factorization
// gave (with the shipped reference's pivots anything else differs visibly):
// inside a panel the 16-row blocks of trsm_dmma_kernel (16 products summed
// from zero, then subtracted), across panels one chain of multiply-adds per
// element in the trailing update's order.  The chain runs through the four
// threads of a row, 32 columns each, one right-hand side behind the other.
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
constexpr int TS_THREADS = 512;   // four threads per row of a tile
constexpr int TS_TLD = TS_B + 1;  // pitch of the diagonal block in shared memory
constexpr int TS_E = TS_B / 4;    // elements of a tile per thread
constexpr int TS_XBUF = TS_B + 8;  // a source's x per right-hand side, padded

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
    const int *rows;  // lower: [panel][n] positions before each panel, by final position
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

template <typename T, bool LOWER, int NR>
__global__ void __launch_bounds__(TS_THREADS, 1) tri_solve_kernel(const TriParams<T> P)
{
    constexpr bool EXACT = LOWER && sizeof(T) == 8;  // the factorization's order of operations
    constexpr int XQ = EXACT ? TS_B + 8 : 1, XB = TS_XBUF * NR;
    // element (row c, right-hand side q) of a source's x: for the chain by
    // right-hand side, padded so that the four threads of a row hit distinct banks
    auto xi = [](int c, int q) { return EXACT ? q * XQ + c + 2 * (c >> 5) : c * NR + q; };
    extern __shared__ __align__(16) unsigned char ts_smem[];
    const int G = gridDim.x, cta = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nblk = P.nblk;
    const int n_own = cta < nblk ? (nblk - cta + G - 1) / G : 0;
    T *Td = reinterpret_cast<T *>(ts_smem);   // [TS_B][TS_TLD], the owned diagonal block solved next
    T *xs = Td + TS_B * TS_TLD;  // [2][TS_XBUF NR]
    T *acc = xs + 2 * XB;                     // [n_own][TS_B][NR]
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

    // solve owned block k (all updates applied) into xs[buf] and x; one warp
    // per right-hand side, lane l holding rows l, l + 32, l + 64, l + 96
    auto solve = [&](int k, int buf) {
        const int p = cta + k * G, r0 = r0_of(p), rows = rows_of(p);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (warp < NR && warp < P.nr) {
            T y[4];
#pragma unroll
            for (int m = 0; m < 4; m++) {
                const int r = 32 * m + lane;
                y[m] = acc[((size_t)k * TS_B + r) * NR + warp];
                if (LOWER && p % P.bpp == 0) y[m] *= sdinv[k * TS_B + r];  // a panel's first block: nothing scaled it yet
            }
#pragma unroll
            for (int mm = 0; mm < 4; mm++) {
                const int mo = LOWER ? mm : 3 - mm;  // the rows being finished
                T s[4];  // EXACT: a 16-column block's products, subtracted together
#pragma unroll 1
                for (int ll = 0; ll < 32; ll += 4) {
                    const int l0 = LOWER ? ll : 28 - ll, c0 = 32 * mo + l0;
                    if (c0 >= rows) continue;
                    // the four columns c0..c0+3 in solve order: e-th is column ce(e)
                    T xv[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) xv[e] = __shfl_sync(0xffffffffu, y[mo], l0 + (LOWER ? e : 3 - e));
#pragma unroll
                    for (int e = 1; e < 4; e++)
#pragma unroll
                        for (int f = 0; f < e; f++) {
                            const int re = c0 + (LOWER ? e : 3 - e), cf = c0 + (LOWER ? f : 3 - f);
                            xv[e] -= Td[re * TS_TLD + cf] * xv[f];
                        }
                    // the other rows; of block mo the lanes beyond the four
#pragma unroll
                    for (int m = 0; m < 4; m++) {
                        if (LOWER ? m < mo : m > mo) continue;
                        // rows after the 16-column block (EXACT): from zero at the block's first columns
                        const bool far = EXACT && (m != mo || (ll < 16 && lane >= 16));
                        T v = y[m];
                        if (far) v = (ll & 15) == 0 ? T(0) : s[m];
                        const T *tr = Td + (32 * m + lane) * TS_TLD + c0;
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            const T t = tr[LOWER ? e : 3 - e];
                            v = fma(far ? t : -t, xv[e], v);
                        }
                        if (far) {
                            s[m] = v;
                            if ((ll & 15) == 12 || c0 + 4 >= rows) y[m] -= v;
                        } else if (m != mo) {
                            y[m] = v;
                        } else {
                            if (LOWER ? lane > l0 + 3 : lane < l0) y[m] = v;
#pragma unroll
                            for (int e = 0; e < 4; e++)
                                if (lane == l0 + (LOWER ? e : 3 - e)) y[m] = xv[e];
                        }
                    }
                }
            }
            unsigned long long *slot = P.xslots + (size_t)r0 * (2 * BS_MAXR);
            T *X = xs + buf * XB;
#pragma unroll
            for (int m = 0; m < 4; m++) {
                const int r = 32 * m + lane;
                if (r < rows) st_stamped(slot + 2 * (r * BS_MAXR + warp), P.epoch, (double)y[m]);
                X[xi(r, warp)] = r < rows ? y[m] : T(0);
            }
#pragma unroll
            for (int m = 0; m < 4; m++) {
                const int r = 32 * m + lane;
                if (r < rows) P.x[(size_t)(r0 + r) * P.ldx + warp] = y[m];
            }
        } else if (warp < NR) {
            for (int r = lane; r < TS_B; r += 32) xs[buf * XB + xi(r, warp)] = T(0);
        }
        __syncthreads();
        if (k + 1 < n_own) prefetch_diag(k + 1);
    };

    // this thread's row of owned block k in source p_src's tile
    const int tr = tid >> 2, part = tid & 3;
    auto tile_row = [&](int k, int p_src) -> int {
        const int p = cta + k * G, r = r0_of(p) + tr;
        if (tr >= rows_of(p)) return -1;
        if (!LOWER || panel_of(p) == panel_of(p_src)) return r;
        return __ldg(P.rows + (size_t)(panel_of(p_src) + 1) * P.n + r);  // its position after the source's panel
    };
    // the thread's 32 columns of the tile's row as v (zero outside): column
    // pairs 8 j + 2 part, 8 j + 2 part + 1 (j = 0..15), of which the four
    // threads of a row read 64 (float: 32) contiguous bytes per load; or
    // (EXACT) columns 32 part .. 32 part + 31
    const bool vec = ((reinterpret_cast<uintptr_t>(P.a) & (2 * sizeof(T) - 1)) == 0) && ((P.ld & 1) == 0) &&
                     (!LOWER || (P.nb & 1) == 0);
    constexpr int CJ = EXACT ? 2 : 8, CP = EXACT ? 32 : 2;  // column of pair j of part: CJ j + CP part
    auto load_tile = [&](int row, int p_src, T (&v)[TS_E]) {
        const int c0 = r0_of(p_src), cols = rows_of(p_src);
        if (row >= 0) {
            const T *u = P.a + (size_t)row * P.ld + c0 + CP * part;
            if (vec && cols == TS_B) {
#pragma unroll
                for (int j = 0; j < TS_E / 2; j++) ts_ld2(u + CJ * j, v[2 * j], v[2 * j + 1]);
            } else {
#pragma unroll
                for (int j = 0; j < TS_E / 2; j++) {
                    const int col = CJ * j + CP * part;
                    v[2 * j] = col < cols ? __ldg(u + CJ * j) : T(0);
                    v[2 * j + 1] = col + 1 < cols ? __ldg(u + CJ * j + 1) : T(0);
                }
            }
        } else {
#pragma unroll
            for (int e = 0; e < TS_E; e++) v[e] = T(0);
        }
    };
    // acc[k] -= tile * X; the first source of the block's own panel finds it
    // updated by all earlier panels and scales it by 1/pivot before
    auto apply_tile = [&](int k, int p_src, const T (&v)[TS_E], const T *X) {
        const int p = cta + k * G;
        const bool own = LOWER && panel_of(p_src) == panel_of(p), live = tr < rows_of(p);
        T *o = acc + ((size_t)k * TS_B + tr) * NR;
        if constexpr (EXACT) {
            if (!own) {
                // the chain: right-hand side q is in part `part` at step q + part
                T a = T(0);
#pragma unroll 1
                for (int step = 0; step < NR + 3; step++) {
                    const int q = step - part;
                    const T in = __shfl_up_sync(0xffffffffu, a, 1);
                    const bool on = q >= 0 && q < NR;
                    const int qc = on ? q : 0;
                    a = part == 0 ? o[qc] : in;
                    const T *xq = X + xi(32 * part, qc);
#pragma unroll
                    for (int g = 0; g < TS_E; g += 8) {  // the trailing update's order within 8 columns
#pragma unroll
                        for (int e = 0; e < 8; e += 2) a = fma(-v[g + e], xq[g + e], a);
#pragma unroll
                        for (int e = 1; e < 8; e += 2) a = fma(-v[g + e], xq[g + e], a);
                    }
                    if (part == 3 && on && live) o[q] = a;
                }
                return;
            }
            const bool scale = p_src % P.bpp == 0;
            const T d = scale ? sdinv[k * TS_B + tr] : T(1);
#pragma unroll 1
            for (int q = 0; q < NR; q++) {
                const T *xq = X + xi(32 * part, q);
                T s0 = T(0), s1 = T(0);
#pragma unroll
                for (int e = 0; e < 16; e++) {
                    s0 = fma(v[e], xq[e], s0);
                    s1 = fma(v[16 + e], xq[16 + e], s1);
                }
                T a = o[q];
                if (scale) a *= d;
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    a -= __shfl_sync(0xffffffffu, s0, (lane & ~3) + e);
                    a -= __shfl_sync(0xffffffffu, s1, (lane & ~3) + e);
                }
                __syncwarp();
                if (part == 0 && live) o[q] = a;
            }
            return;
        }
        T s[NR];
#pragma unroll
        for (int q = 0; q < NR; q++) s[q] = T(0);
#pragma unroll
        for (int e = 0; e < TS_E; e++) {
            const T *xr = X + xi(8 * (e >> 1) + 2 * part + (e & 1), 0);
#pragma unroll
            for (int q = 0; q < NR; q++) s[q] += v[e] * xr[q];
        }
#pragma unroll
        for (int q = 0; q < NR; q++) {
            s[q] += __shfl_xor_sync(0xffffffffu, s[q], 1);
            s[q] += __shfl_xor_sync(0xffffffffu, s[q], 2);
        }
        if (part == 0 && live) {
            const bool scale = own && p_src % P.bpp == 0;
            const T d = LOWER && scale ? sdinv[k * TS_B + tr] : T(1);
#pragma unroll
            for (int q = 0; q < NR; q++) o[q] = (scale ? o[q] * d : o[q]) - s[q];
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
    int row = next < n_own ? tile_row(next, 0) : -1;
    for (int p_src = 0; p_src < nblk; p_src++) {
        const int buf = p_src & 1;
        T *X = xs + buf * XB;
        const int k_first = next;
        T v[TS_E];
        if (k_first < n_own) {
            load_tile(row, p_src, v);
            if (p_src + 1 < nblk) row = tile_row(k_first, p_src + 1);
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
                if (e >= TS_B * NR) continue;
                if (r < rows && q < P.nr)
                    todo |= 1u << u;
                else
                    X[xi(r, q)] = T(0);
            }
            for (unsigned round = 1;; round++) {
#pragma unroll
                for (int u = 0; u < EPT; u++) {
                    if (!((todo >> u) & 1u)) continue;
                    const int e = tid + u * TS_THREADS, r = e / NR, q = e % NR;
                    unsigned long long hi, lo;
                    ld_pair(slot + 2 * (r * BS_MAXR + q), hi, lo);
                    if (stamped(hi, P.epoch) && stamped(lo, P.epoch)) {
                        X[xi(r, q)] = (T)unstamp(hi, lo);
                        todo &= ~(1u << u);
                    }
                }
                if (__syncthreads_and(todo == 0)) break;
                const bool late = (round & 63u) == 0 && tid == 0 &&
                                  (*(volatile int *)&P.status[1] != 0 || globaltimer_ns() - t0 > WAIT_LIMIT_NS);
                if ((round & 63u) == 0 && __syncthreads_or(late)) {
                    if (tid == 0 && *(volatile int *)&P.status[1] == 0) record_error(P.status, ERR_BARRIER_TIMEOUT, 6);
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
                if (next < n_own && p_src + 1 < nblk) row = tile_row(next, p_src + 1);
            }
        }
        for (int k = k_first + 1; k < n_own; k++) {
            load_tile(tile_row(k, p_src), p_src, v);
            apply_tile(k, p_src, v, X);
        }
        __syncthreads();  // X (this buffer) is overwritten two sources later
    }
}

template <typename T, bool LOWER, int NR>
static cudaError_t ts_launch(TriParams<T> P, cudaStream_t st, bool *used)
{
    *used = false;
    int dev = 0, sms = 148;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    const int G = P.nblk < sms ? P.nblk : sms, own = (P.nblk + G - 1) / G;
    const size_t smem = ((size_t)TS_B * TS_TLD + 2 * TS_XBUF * NR + (size_t)own * TS_B * (NR + (LOWER ? 1 : 0))) * sizeof(T);
    if (smem > 220 * 1024) return cudaSuccess;  // too many blocks per CTA: the caller's other way
    auto kern = tri_solve_kernel<T, LOWER, NR>;
    if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024)) != cudaSuccess) return e;
    void *args[] = {&P};
    count_launch();
    e = cudaLaunchCooperativeKernel((const void *)kern, dim3(G), dim3(TS_THREADS), args, smem, st);
    if (e == cudaSuccess) *used = true;
    return e;
}

// up to BS_MAXR right-hand sides, padded to the next of 1, 2, 4, 8
template <typename T, bool LOWER>
static cudaError_t ts_any(TriParams<T> P, const BsBuffers &bs, cudaStream_t st, bool *used)
{
    *used = false;
    if (P.n > bs.cap_rows) return cudaSuccess;
    P.xslots = bs.xslots;
    P.status = bs.status;
    P.epoch = ++*bs.epoch;
    if (P.epoch == 0) P.epoch = ++*bs.epoch;
    if (P.nr == 1) return ts_launch<T, LOWER, 1>(P, st, used);
    if (P.nr == 2) return ts_launch<T, LOWER, 2>(P, st, used);
    if (P.nr <= 4) return ts_launch<T, LOWER, 4>(P, st, used);
    return ts_launch<T, LOWER, 8>(P, st, used);
}

template <typename T>
static cudaError_t upper_t(const T *a, long ld, int n, int nrhs, const T *y, long ldy, T *x, long ldx,
                           const BsBuffers &bs, cudaStream_t st, bool *used)
{
    *used = false;
    for (int c0 = 0; c0 < nrhs; c0 += BS_MAXR) {
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
        P.nr = nrhs - c0 < BS_MAXR ? nrhs - c0 : BS_MAXR;
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

template <typename T>
static cudaError_t lower_t(const T *a, long ld, int n, int nb, const int *rows, const T *dinv, const T *b, long ldb,
                           int nrhs, T *y, long ldy, const BsBuffers &bs, cudaStream_t st, bool *used)
{
    *used = false;
    if (nrhs > BS_MAXR) return cudaErrorInvalidValue;
    TriParams<T> P{};
    P.a = a;
    P.ld = ld;
    P.n = n;
    P.nb = nb;
    P.bpp = (nb + TS_B - 1) / TS_B;
    const int npan = (n + nb - 1) / nb, last = n - (npan - 1) * nb;
    P.nblk = (npan - 1) * P.bpp + (last + TS_B - 1) / TS_B;
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

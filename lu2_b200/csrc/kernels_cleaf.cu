// kernels_cleaf.cu -- the panel leaf on one thread-block cluster: LU with
// partial pivoting of a slab of up to 64 columns whose rows live in the
// registers of at most 16 CTAs.
//
// Reference behaviour (telmin/lu2): column_decomposition, lu2tlib.c:1041-1066
// inside the slab recursion lu2tlib.c:1095-1128; pivot search cblas_idamax
// (first max of |a|), lu2tlib.c:42-52; the pivot row is scaled by 1/pivot in
// every column but the diagonal, lu2tlib.c:1057-1059.  Per element the same
// operations in the same order as leaf_kernel (kernels_leaf.cu).
//
// What bounds it: one pivot decision per column, a chain of dependent steps
// that no amount of bandwidth shortens.  Over the whole grid that chain costs
// four trips through L2 per column (kernels_leaf.cu: 3.6-4.6 us); inside a
// cluster it is one CTA barrier and one trip through distributed shared
// memory.  So:
//  * a thread holds R whole rows in registers; no row ever moves.  Each row
//    carries its current position in the matrix (`pos`): an exchange c <-> p
//    is two threads changing their positions, and a row is written back to
//    its last position at the end.
//  * the registers rotate: eliminating column j writes r[j+1] - l u[j+1] into
//    r[j], so the loop over columns is one rolled body (its current column is
//    always r[0]); the multiplier l goes to the row's shared-memory slot, which
//    is stored to the matrix at the end.
//  * the candidate of a warp is found with redux.sync on the bits of |a|
//    (the upper word decides except in ties), its row goes to shared memory
//    before the column's one CTA barrier, and after it the CTA's candidate
//    row, already scaled by 1/pivot, is sent to every CTA of the cluster with
//    st.async, which completes an mbarrier there.  Every warp then picks the
//    winner from the CTAs' candidates by itself.
// Messages and candidate rows are double-buffered by column parity: a CTA can
// be one column ahead of another at most, since it needs that CTA's message of
// a column to leave it, and each buffer's readers have passed the next
// column's CTA barrier before their CTA sends that column's message.
//
// Every wait is bounded: when one gives up, the CTA records the error and
// leaves the loop at its next barrier; the others find the error word and do
// the same.  No CTA exits before all have arrived at the last cluster barrier.
#include <atomic>
#include <climits>

#include "lu2gpu_internal.cuh"

namespace lu2gpu {

template <typename T>
struct CLeafParams {
    T *a;
    long ld;
    int n, c0, w, rpc, mode, goff;  // rpc: rows per CTA
    int *ipiv;
    T *dinv;
    int *status;
    unsigned long long wait_ns;
    int withhold;
};

template <typename T, int W, int R, int TPB>
struct CLeafCfg {
    static constexpr int NW = TPB / 32;
    static constexpr int VEC = 16 / (int)sizeof(T);
    static constexpr int PITCH = W + VEC;  // a slot's 16-byte accesses by consecutive rows hit distinct banks
    static constexpr int ROWS = R * TPB;   // rows a CTA holds
    static constexpr int PIECES = 1 + W / VEC;
    static constexpr int MSG = 16 * PIECES;  // header (key, position), then the row
    static constexpr int MAXC = 16;
    static constexpr size_t O_SLAB = 0;
    static constexpr size_t O_WROW = O_SLAB + (size_t)ROWS * PITCH * sizeof(T);
    static constexpr size_t O_MSG = O_WROW + (size_t)2 * NW * W * sizeof(T);
    static constexpr size_t O_U = O_MSG + (size_t)2 * MAXC * MSG;  // one CTA: each warp's scaled pivot row
    static constexpr size_t O_POS = O_U + (size_t)NW * W * sizeof(T);
    static constexpr size_t SMEM = O_POS + (size_t)ROWS * sizeof(int);
};

__device__ __forceinline__ unsigned cl_smem(const void *p)
{
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

// Pivot candidates order as (key, then lower position): key 0 = not a
// candidate, 1 = row c holding a NaN (taken when nothing else is left: such a
// column keeps its row), else the bits of |v| + 2 -- for float in the upper word.
__device__ __forceinline__ unsigned long long cl_key(double v, bool at_c)
{
    return v == v ? (unsigned long long)__double_as_longlong(fabs(v)) + 2ull : (at_c ? 1ull : 0ull);
}
__device__ __forceinline__ unsigned long long cl_key(float v, bool at_c)
{
    return v == v ? (unsigned long long)(__float_as_uint(fabsf(v)) + 2u) << 32 : (at_c ? 1ull : 0ull);
}

// the lane holding the warp's best candidate
__device__ __forceinline__ int cl_winner(unsigned long long key, int pos)
{
    const unsigned full = 0xffffffffu, hi = (unsigned)(key >> 32), lo = (unsigned)key;
    const unsigned mh = __reduce_max_sync(full, hi);
    bool in = hi == mh;
    unsigned b = __ballot_sync(full, in);
    if (b & (b - 1)) {
        const unsigned ml = __reduce_max_sync(full, in ? lo : 0u);
        in = in && lo == ml;
        b = __ballot_sync(full, in);
        if (b & (b - 1)) {
            const unsigned mp = __reduce_min_sync(full, in ? (unsigned)pos : 0xffffffffu);
            b = __ballot_sync(full, in && (unsigned)pos == mp);
        }
    }
    return __ffs(b) - 1;
}

__device__ __forceinline__ double cl_fnma(double l, double u, double x) { return fma(-l, u, x); }
__device__ __forceinline__ float cl_fnma(float l, float u, float x) { return fmaf(-l, u, x); }

// one 16-byte piece of a row
__device__ __forceinline__ void cl_ld16(const void *p, double (&v)[2])
{
    const double2 x = *reinterpret_cast<const double2 *>(p);
    v[0] = x.x;
    v[1] = x.y;
}
__device__ __forceinline__ void cl_ld16(const void *p, float (&v)[4])
{
    const float4 x = *reinterpret_cast<const float4 *>(p);
    v[0] = x.x;
    v[1] = x.y;
    v[2] = x.z;
    v[3] = x.w;
}
__device__ __forceinline__ void cl_st16(void *p, const double (&v)[2])
{
    *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]);
}
__device__ __forceinline__ void cl_st16(void *p, const float (&v)[4])
{
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void cl_bits(const double (&v)[2], unsigned long long &a, unsigned long long &b)
{
    a = (unsigned long long)__double_as_longlong(v[0]);
    b = (unsigned long long)__double_as_longlong(v[1]);
}
__device__ __forceinline__ void cl_bits(const float (&v)[4], unsigned long long &a, unsigned long long &b)
{
    a = __float_as_uint(v[0]) | (unsigned long long)__float_as_uint(v[1]) << 32;
    b = __float_as_uint(v[2]) | (unsigned long long)__float_as_uint(v[3]) << 32;
}

// A row travels as its columns after the current one, then the current one:
// element j < W - 1 is column j + 1 of the rotated row, element W - 1 the pivot.
template <typename T, int W, int R, int TPB>
__global__ void __launch_bounds__(TPB, 1) cluster_leaf_kernel(const CLeafParams<T> P)
{
    using C = CLeafCfg<T, W, R, TPB>;
    constexpr int NW = C::NW, VEC = C::VEC, PITCH = C::PITCH, PIECES = C::PIECES, MSG = C::MSG;
    extern __shared__ __align__(16) unsigned char cl_dyn[];
    T *slab = reinterpret_cast<T *>(cl_dyn + C::O_SLAB);
    T *wrow = reinterpret_cast<T *>(cl_dyn + C::O_WROW);
    unsigned char *msg = cl_dyn + C::O_MSG;
    int *spos = reinterpret_cast<int *>(cl_dyn + C::O_POS);
    __shared__ unsigned long long s_key[2][NW];
    __shared__ int s_pos[2][NW];
    __shared__ __align__(8) unsigned long long s_bar[2];
    __shared__ T s_inv[W];
    __shared__ int s_fail[2];  // by column parity: set in a column's wait, read after the next column's barrier
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int CL = gridDim.x, rank = blockIdx.x;  // one cluster per launch
    const int c0 = P.c0, w = P.w;
    const int rb = c0 + rank * P.rpc, nr = max(0, min(P.rpc, P.n - rb));

    // the CTA's rows into their slots, 16 bytes per copy (zeros past column w)
    constexpr int CPR = W / VEC;  // copies per row
    for (int q = tid; q < nr * CPR; q += TPB) {
        const int lr = q / CPR, ch = q % CPR;
        const int have = min(VEC, max(0, w - ch * VEC)) * (int)sizeof(T);
        const T *src = P.a + (size_t)(rb + lr) * P.ld + c0 + (have ? ch * VEC : 0);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(cl_smem(slab + lr * PITCH + ch * VEC)),
                     "l"(src), "r"(have)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (tid == 0) {
        s_fail[0] = *(volatile int *)&P.status[1] != 0;  // an earlier wait of this call gave up: nothing to do
        s_fail[1] = 0;
        for (int b = 0; b < 2; b++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(cl_smem(&s_bar[b])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // the barriers exist before any CTA sends to them
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    __syncthreads();

    T r[R][W];
    T ls[R];     // the multiplier the reference's pivot searches look at
    int pos[R];  // the row's current position (rows of the view); -1: no row
#pragma unroll
    for (int k = 0; k < R; k++) {
        const int lr = tid + k * TPB;
        pos[k] = lr < nr ? rb + lr : -1;
        ls[k] = T(0);
#pragma unroll
        for (int j = 0; j < W; j += VEC) {
            T v[VEC];
            if (lr < nr) {
                cl_ld16(slab + lr * PITCH + j, v);
            } else {
#pragma unroll
                for (int e = 0; e < VEC; e++) v[e] = T(0);
            }
#pragma unroll
            for (int e = 0; e < VEC; e++) r[k][j + e] = v[e];
        }
    }

#pragma unroll 1
    for (int ip = 0; ip < w; ip++) {
        const int c = c0 + ip, par = ip & 1, rem = w - ip;
        const bool use_ls = ip > 0 && ((P.mode == PIVOT_REF && ((c + P.goff) & 1)) ||  // lu2tlib.c:1052
                                       P.mode == PIVOT_REF_FIRST);
        // this thread's candidate, the warp's, the CTA's
        unsigned long long key = 0;
        int kp = INT_MAX, kr = 0;
#pragma unroll
        for (int k = 0; k < R; k++) {
            const unsigned long long kk = pos[k] >= c ? cl_key(use_ls ? ls[k] : r[k][0], pos[k] == c) : 0ull;
            if (kk > key || (kk == key && kk != 0 && pos[k] < kp)) {
                key = kk;
                kp = pos[k];
                kr = k;
            }
        }
        if (lane == cl_winner(key, kp)) {
            T *dst = wrow + (par * NW + warp) * W;
#pragma unroll
            for (int k = 0; k < R; k++)
                if (R == 1 || kr == k) {
#pragma unroll
                    for (int j = 0; j < W; j += VEC) {
                        T v[VEC];
#pragma unroll
                        for (int e = 0; e < VEC; e++) v[e] = r[k][(j + e + 1) % W];
                        if (j < rem || j + VEC == W) cl_st16(dst + j, v);
                    }
                }
            s_key[par][warp] = key;
            s_pos[par][warp] = kp;
        }
        __syncthreads();
        if (s_fail[par]) break;
        unsigned long long ck = lane < NW ? s_key[par][lane] : 0ull;
        int cp = lane < NW ? s_pos[par][lane] : INT_MAX;
        const int ww = cl_winner(ck, cp);
        ck = __shfl_sync(0xffffffffu, ck, ww);
        cp = __shfl_sync(0xffffffffu, cp, ww);
        const T *row = wrow + (par * NW + ww) * W;
        const T *u;
        int p = cp;
        if (CL == 1) {
            const T d = row[W - 1], inv = d == T(0) ? T(1) : T(1) / d;
            T *mine = reinterpret_cast<T *>(cl_dyn + C::O_U) + warp * W;
            if (lane < CPR) {
                T v[VEC];
                cl_ld16(row + lane * VEC, v);
#pragma unroll
                for (int e = 0; e < VEC; e++)
                    if (lane * VEC + e != W - 1) v[e] *= inv;
                cl_st16(mine + lane * VEC, v);
            }
            __syncwarp();
            u = mine;
        } else {
            const T d = row[W - 1], inv = d == T(0) ? T(1) : T(1) / d;
            const unsigned bar = cl_smem(&s_bar[par]);
            if (tid == 0)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(CL * MSG)
                             : "memory");
            if (rank != P.withhold)
#pragma unroll 1
                for (int q = tid; q < CL * PIECES; q += TPB) {
                    const int to = q / PIECES, piece = q - to * PIECES;
                    unsigned long long x0 = ck, x1 = (unsigned)cp;
                    if (piece > 0) {
                        T v[VEC];
                        cl_ld16(row + (piece - 1) * VEC, v);
#pragma unroll
                        for (int e = 0; e < VEC; e++)
                            if ((piece - 1) * VEC + e != W - 1) v[e] *= inv;
                        cl_bits(v, x0, x1);
                    }
                    unsigned dst, rbar;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                                 : "=r"(dst)
                                 : "r"(cl_smem(msg + (par * C::MAXC + rank) * MSG + piece * 16)), "r"(to));
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rbar) : "r"(bar), "r"(to));
                    asm volatile(
                        "st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(dst),
                        "l"(x0), "l"(x1), "r"(rbar)
                        : "memory");
                }
            // every CTA's candidate of this column
            const unsigned parity = (unsigned)(ip >> 1) & 1u;
            unsigned long long t0 = 0;
            for (unsigned spins = 1;; spins++) {
                unsigned ok;
                asm volatile(
                    "{\n\t.reg .pred P1;\n\t"
                    "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P1, [%1], %2;\n\t"
                    "selp.b32 %0, 1, 0, P1;\n\t}"
                    : "=r"(ok)
                    : "r"(bar), "r"(parity)
                    : "memory");
                if (ok) break;
                if ((spins & 15u) == 0) {
                    const unsigned long long now = globaltimer_ns();
                    if (t0 == 0) t0 = now;
                    if (*(volatile int *)&P.status[1] != 0 || now - t0 > P.wait_ns) {
                        if (*(volatile int *)&P.status[1] == 0) record_error(P.status, ERR_BARRIER_TIMEOUT, 1);
                        *(volatile int *)&s_fail[par ^ 1] = 1;  // the CTA leaves at its next barrier
                        break;
                    }
                }
            }
            __syncwarp();
            const unsigned char *m0 = msg + (size_t)par * C::MAXC * MSG;
            ck = 0;
            cp = INT_MAX;
            if (lane < CL) {
                ck = *reinterpret_cast<const unsigned long long *>(m0 + lane * MSG);
                cp = *reinterpret_cast<const int *>(m0 + lane * MSG + 8);
            }
            const int wc = cl_winner(ck, cp);
            p = __shfl_sync(0xffffffffu, cp, wc);
            u = reinterpret_cast<const T *>(m0 + wc * MSG + 16);
        }

        const T d = u[W - 1];
        const bool zero = d == T(0);
        // row c of the factors from column c on, the pivot and its reciprocal
        if (warp == NW - 1) {
            const T inv = zero ? T(1) : T(1) / d;
            if (lane == 0) s_inv[ip] = inv;
            if (rank == 0) {
                T *dst = P.a + (size_t)c * P.ld + c;
                for (int j = lane; j < rem; j += 32) dst[j] = j == 0 ? d : u[j - 1];
                if (lane == 0) {
                    P.ipiv[c] = p + P.goff;
                    P.dinv[c] = inv;
                    if (zero) atomicMin(&P.status[0], c + 1);
                }
            }
        }
        T l[R];
#pragma unroll
        for (int k = 0; k < R; k++) {
            l[k] = r[k][0];
            if (pos[k] >= c) {
                if (pos[k] == p) {
                    pos[k] = c;
                } else {
                    if (pos[k] == c) pos[k] = p;
                    slab[(tid + k * TPB) * PITCH + ip] = l[k];
                }
            }
            if (P.mode == PIVOT_REF || ip == 0) ls[k] = l[k];
        }
        // rank-1 update, rotating; rows that are done compute values nobody reads
        constexpr int GW = W < 8 ? W : 8;
#pragma unroll
        for (int g = 0; g < W; g += GW) {
            if (g >= rem) break;
            T ug[GW];
#pragma unroll
            for (int j = 0; j < GW; j += VEC) {
                T v[VEC];
                cl_ld16(u + g + j, v);
#pragma unroll
                for (int e = 0; e < VEC; e++) ug[j + e] = v[e];
            }
            if (!zero) {
#pragma unroll
                for (int k = 0; k < R; k++)
#pragma unroll
                    for (int j = 0; j < GW; j++)
                        if (g + j + 1 < W) r[k][g + j] = cl_fnma(l[k], ug[j], r[k][g + j + 1]);
            } else {
#pragma unroll
                for (int k = 0; k < R; k++)
#pragma unroll
                    for (int j = 0; j < GW; j++)
                        if (g + j + 1 < W) r[k][g + j] = r[k][g + j + 1];
            }
        }
    }
    __syncthreads();
    const bool fail = (s_fail[0] | s_fail[1]) != 0;
    if (!fail) {
        // the multipliers to the rows' last positions; a pivot row's are
        // scaled by its 1/pivot like the rest of it, and its columns from its
        // own on are in the matrix already
#pragma unroll
        for (int k = 0; k < R; k++)
            if (tid + k * TPB < nr) spos[tid + k * TPB] = pos[k];
        __syncthreads();
        for (int q = tid; q < nr * CPR; q += TPB) {
            const int lr = q / CPR, ch = q % CPR;
            const int at = spos[lr], have = min(w, at - c0) - ch * VEC;
            if (have <= 0) continue;
            T *dst = P.a + (size_t)at * P.ld + c0 + ch * VEC;
            T v[VEC];
            cl_ld16(slab + lr * PITCH + ch * VEC, v);
            if (at < c0 + w) {
#pragma unroll
                for (int e = 0; e < VEC; e++) v[e] *= s_inv[at - c0];
            }
            if (have >= VEC) {
                cl_st16(dst, v);
            } else {
#pragma unroll
                for (int e = 0; e < VEC; e++)
                    if (e < have) dst[e] = v[e];
            }
        }
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// ---------------------------------------------------------------------------
// The widest slab one cluster of 16 holds in registers, by rows (128 registers
// a thread with 512 threads, 255 with 256):
//   FP64: 64 columns to 4096 rows, 32 to 8192, 16 to 16384
//   FP32: 64 columns to 8192 rows, 32 to 16384, 16 to 32768
// A wider leaf replaces whole levels of the panel recursion (four launches
// each) by rank-1 steps in registers.  Taller panels go to leaf_kernel.
template <typename T, int W>
struct CLeafPick;
template <>
struct CLeafPick<double, 64> {
    static constexpr int R = 1, TPB = 256;
};
template <>
struct CLeafPick<double, 32> {
    static constexpr int R = 1, TPB = 512;
};
template <>
struct CLeafPick<double, 16> {
    static constexpr int R = 2, TPB = 512;
};
template <>
struct CLeafPick<float, 64> {
    static constexpr int R = 1, TPB = 512;
};
template <>
struct CLeafPick<float, 32> {
    static constexpr int R = 2, TPB = 512;
};
template <>
struct CLeafPick<float, 16> {
    static constexpr int R = 4, TPB = 512;
};

template <typename T, int W>
static constexpr int cl_rows()
{
    return 16 * CLeafPick<T, W>::R * CLeafPick<T, W>::TPB;
}

// shared memory and cluster size limits of one instance; true when a cluster of 16 can be resident
template <typename T, int W>
static bool cl_prepare()
{
    using K = CLeafPick<T, W>;
    using C = CLeafCfg<T, W, K::R, K::TPB>;
    auto kern = cluster_leaf_kernel<T, W, K::R, K::TPB>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
        return false;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(K::TPB);
    cfg.dynamicSmemBytes = C::SMEM;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {16, 1, 1};
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int clusters = 0;
    return cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) == cudaSuccess && clusters >= 1;
}

// whether the current device takes the cluster leaf (looked up once per device)
static bool cl_device_ok()
{
    static std::atomic<signed char> known[128];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 128) return false;
    signed char k = known[dev].load();
    if (k == 0) {
        k = cl_prepare<double, 64>() && cl_prepare<double, 32>() && cl_prepare<double, 16>() &&
                    cl_prepare<float, 64>() && cl_prepare<float, 32>() && cl_prepare<float, 16>()
                ? 1
                : -1;
        cudaGetLastError();
        known[dev].store(k);
    }
    return k > 0;
}

template <typename T>
static int cl_width(int rows, int max_ctas)
{
    if (rows <= 0 || max_ctas < 16 || !cl_device_ok()) return 0;
    if (rows <= cl_rows<T, 64>()) return 64;
    if (rows <= cl_rows<T, 32>()) return 32;
    return rows <= cl_rows<T, 16>() ? 16 : 0;
}

int leaf_width(int rows, size_t tsize, int max_ctas)
{
    const int k = tsize == sizeof(double) ? cl_width<double>(rows, max_ctas) : cl_width<float>(rows, max_ctas);
    return k > 16 ? k : 16;
}

template <typename T, int W>
static cudaError_t cl_launch_w(CLeafParams<T> P, cudaStream_t st)
{
    using K = CLeafPick<T, W>;
    using C = CLeafCfg<T, W, K::R, K::TPB>;
    const int rows = P.n - P.c0;
    int cl = 1;
    while (cl < 16 && cl * C::ROWS < rows) cl *= 2;
    P.rpc = (rows + cl - 1) / cl;
    if (P.rpc > C::ROWS) return cudaErrorInvalidConfiguration;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)cl);
    cfg.blockDim = dim3(K::TPB);
    cfg.dynamicSmemBytes = C::SMEM;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {(unsigned)cl, 1, 1};
    cfg.attrs = at;
    cfg.numAttrs = 1;
    count_launch();
    return cudaLaunchKernelEx(&cfg, cluster_leaf_kernel<T, W, K::R, K::TPB>, P);
}

template <typename T>
static cudaError_t launch_leaf_cluster_t(T *a, long ld, int n, int c0, int w, int mode, int goff, int *ipiv, T *dinv,
                                         const LeafBuffers &buf, int *status, int max_ctas, cudaStream_t st,
                                         bool *used)
{
    *used = false;
    const int width = cl_width<T>(n - c0, max_ctas);
    constexpr int VEC = 16 / (int)sizeof(T);
    // 16-byte copies of row segments
    if (w <= 0 || w > width || (reinterpret_cast<uintptr_t>(a) & 15) || ld % VEC || c0 % VEC) return cudaSuccess;
    *used = true;
    const CLeafParams<T> P{a, ld, n, c0, w, 0, mode, goff, ipiv, dinv, status, buf.wait_ns, buf.withhold};
    if (w <= 16) return cl_launch_w<T, 16>(P, st);
    return w <= 32 ? cl_launch_w<T, 32>(P, st) : cl_launch_w<T, 64>(P, st);
}

cudaError_t launch_leaf_cluster(double *a, long ld, int n, int c0, int w, int mode, int goff, int *ipiv, double *dinv,
                                const LeafBuffers &buf, int *status, int max_ctas, cudaStream_t st, bool *used)
{
    return launch_leaf_cluster_t(a, ld, n, c0, w, mode, goff, ipiv, dinv, buf, status, max_ctas, st, used);
}

cudaError_t launch_leaf_cluster(float *a, long ld, int n, int c0, int w, int mode, int goff, int *ipiv, float *dinv,
                                const LeafBuffers &buf, int *status, int max_ctas, cudaStream_t st, bool *used)
{
    return launch_leaf_cluster_t(a, ld, n, c0, w, mode, goff, ipiv, dinv, buf, status, max_ctas, st, used);
}

}  // namespace lu2gpu

// kernels_cleaf.cu -- the panel leaf on one thread-block cluster: LU with
// partial pivoting of a slab of up to 64 columns whose rows live in the shared
// memory of at most 16 CTAs.
//
// Reference behaviour (telmin/lu2): column_decomposition, lu2tlib.c:1041-1066
// inside the slab recursion lu2tlib.c:1095-1128; pivot search cblas_idamax
// (first max of |a|), lu2tlib.c:42-52; the pivot row is scaled by 1/pivot in
// every column but the diagonal, lu2tlib.c:1057-1059.  Per element the
// operations of leaf_kernel (kernels_leaf.cu) in the same order, but for the
// sums of 8 products below.
//
// What bounds it: one pivot decision per column, a chain of dependent steps
// that no amount of bandwidth shortens, and the instructions that every warp
// of a CTA spends on it.  Over the whole grid that chain costs four trips
// through L2 per column (kernels_leaf.cu: 3.6-4.6 us); inside a cluster it is
// two CTA barriers and one trip through distributed shared memory.  So:
//  * the slab lives in the CTAs' shared memory and is factored in blocks of 8
//    columns, each thread holding the 8 columns of its RT rows in registers.
//    The registers rotate (eliminating a column writes r[j+1] - l u[j+1] into
//    r[j]), so the 8 columns are one rolled loop, small enough for the
//    instruction cache.  A pivot decision then concerns 8 columns: its row is
//    written by one lane in 5 shared stores and travels as 5 pieces of 16
//    bytes.  (Rows of all 64 columns in registers, searched, scaled, sent and
//    updated whole at every column, took 1.14 us a column on one CTA and 1.66
//    on 16.)
//  * no row ever moves: each carries its current position in the matrix
//    (`pos`), an exchange c <-> p is two rows changing their positions, and a
//    row is written back to its last one at the end.
//  * a warp's candidate is found with redux.sync on the bits of |a| (the upper
//    word decides except in ties), the CTA's from the warps' after one
//    barrier; its owner puts the row, scaled by 1/pivot, into shared memory,
//    from where after a second barrier it goes to every CTA of the cluster with
//    st.async, which completes an mbarrier there.  Every warp then picks the
//    winner from the CTAs' candidates by itself.  (Sending the candidates' keys
//    first and the winner's row alone in a second trip measured 1000-1300
//    cycles a column against 750-1100 for the one trip.)
//  * the winner's CTA sends the rest of the row, unchanged since the block
//    began, to every CTA on a second mbarrier, beside the next columns.  After
//    the 8 columns every CTA finishes the 8 pivot rows right of the block by
//    itself (one thread per column, the same multiply-adds in the same order)
//    and subtracts their products from its rows: FP64 on the tensor pipe
//    (mma.sync m16n8k8, the 8 products summed first), FP32 on the CUDA cores.
// Messages are double-buffered by column parity: a CTA can be one column ahead
// of another at most, since it needs that CTA's message of a column to leave
// it, and a buffer's readers have passed the next column's CTA barriers before
// their CTA sends that column's message.
//
// Every wait is bounded: when one gives up, the CTA records the error and
// leaves the loop at its next barrier; the others find the error word and do
// the same.  No CTA exits before all have arrived at the last cluster barrier,
// and one that gave up stays a little longer, for what is still on its way to it.
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

constexpr int CL_TPB = 256, CL_NW = CL_TPB / 32;  // threads with rows
constexpr int CL_HELP = 128;  // helpers: store and send the decided rows beside the next column's search
constexpr int CL_ALL = CL_TPB + CL_HELP;
constexpr int CL_B = 8;      // columns of a block
constexpr int CL_MAXC = 16;  // CTAs of a cluster
constexpr unsigned long long CL_LINGER_NS = 50000;  // that a CTA stays after a failed wait

template <typename T, int W, int RT>
struct CLeafCfg {
    static constexpr int VEC = 16 / (int)sizeof(T);
    static constexpr int PITCH = W + VEC;      // 16-byte accesses of consecutive rows fall on distinct banks
    static constexpr int ROWS = RT * CL_TPB;   // rows a CTA holds
    static constexpr int MSG = 16 + CL_B * (int)sizeof(T);  // header (key, position, row), the row's 8 columns
    static constexpr int PIECES = MSG / 16;
    static constexpr int UP = W + 4;           // pitch of the finished pivot rows: B fragments on distinct banks
    static constexpr int XP = W + VEC;         // pitch of the received pivot rows
    static constexpr size_t O_SLAB = 0;
    static constexpr size_t O_U = O_SLAB + (size_t)ROWS * PITCH * sizeof(T);
    static constexpr size_t O_X = O_U + (size_t)CL_B * UP * sizeof(T);
    static constexpr size_t O_MSG = O_X + (size_t)CL_B * XP * sizeof(T);
    static constexpr size_t O_POS = O_MSG + (size_t)2 * CL_MAXC * MSG;
    static constexpr size_t SMEM = O_POS + (size_t)ROWS * sizeof(int);
    static_assert(O_X % 16 == 0 && O_MSG % 16 == 0 && MSG % 16 == 0, "16-byte pieces");
};

__device__ __forceinline__ unsigned cl_smem(const void *p)
{
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

// Pivot candidates order as (key, then lower position): key 0 = not a
// candidate, 1 = row c holding a NaN (taken when nothing else is left: such a
// column keeps its row), else the bits of |v| with 2 added to the upper word.
// A float's key is its upper word alone.  (Integer tests: a 64-bit floating
// comparison costs the chain 20 cycles.)
__device__ __forceinline__ unsigned long long cl_key(double v, bool act, bool at_c)
{
    const unsigned hi = (unsigned)__double2hiint(v) & 0x7fffffffu, lo = (unsigned)__double2loint(v);
    const bool nan = (hi > 0x7ff00000u) | ((hi == 0x7ff00000u) & (lo != 0u));
    const unsigned kh = act ? (nan ? (unsigned)at_c : hi + 2u) : 0u, kl = act & !nan ? lo : 0u;
    return (unsigned long long)kh << 32 | kl;
}
__device__ __forceinline__ unsigned long long cl_key(float v, bool act, bool at_c)
{
    const unsigned b = __float_as_uint(v) & 0x7fffffffu;
    return (unsigned long long)(act ? (b > 0x7f800000u ? (unsigned)at_c : b + 2u) : 0u) << 32;
}
__device__ __forceinline__ bool cl_zero(double v) { return ((unsigned long long)__double_as_longlong(v) << 1) == 0; }
__device__ __forceinline__ bool cl_zero(float v) { return (__float_as_uint(v) << 1) == 0; }

// the lane holding the warp's best candidate (some lane when there is none:
// warps without rows went through the tie path, 56.6 -> 53.7 us on 200 rows)
__device__ __forceinline__ int cl_winner(unsigned long long key, int pos, int lane)
{
    const unsigned full = 0xffffffffu, hi = (unsigned)(key >> 32), lo = (unsigned)key;
    const unsigned mh = __reduce_max_sync(full, hi);
    bool in = hi == mh;
    const unsigned b = __ballot_sync(full, in);
    unsigned win = __reduce_min_sync(full, in ? (unsigned)lane : 31u);
    if ((b & (b - 1)) && mh) {  // a tie in the upper word
        const unsigned ml = __reduce_max_sync(full, in ? lo : 0u);
        in = in && lo == ml;
        const unsigned mp = __reduce_min_sync(full, in ? (unsigned)pos : 0xffffffffu);
        win = __reduce_min_sync(full, in && (unsigned)pos == mp ? (unsigned)lane : 31u);
    }
    return (int)win;
}

__device__ __forceinline__ double cl_fnma(double l, double u, double x) { return fma(-l, u, x); }
__device__ __forceinline__ float cl_fnma(float l, float u, float x) { return fmaf(-l, u, x); }

// shared memory by its 32-bit address: 16-byte pieces of a row, headers, words
__device__ __forceinline__ void cl_ld16(unsigned p, double (&v)[2])
{
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "r"(p));
}
__device__ __forceinline__ void cl_ld16(unsigned p, float (&v)[4])
{
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
                 : "r"(p));
}
__device__ __forceinline__ void cl_st16(unsigned p, const double (&v)[2])
{
    asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(p), "d"(v[0]), "d"(v[1]) : "memory");
}
__device__ __forceinline__ void cl_st16(unsigned p, const float (&v)[4])
{
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3])
                 : "memory");
}
__device__ __forceinline__ void cl_put16(double *p, const double (&v)[2])
{
    *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]);
}
__device__ __forceinline__ void cl_put16(float *p, const float (&v)[4])
{
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void cl_st1(unsigned p, double v)
{
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(p), "d"(v) : "memory");
}
__device__ __forceinline__ void cl_st1(unsigned p, float v)
{
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(p), "f"(v) : "memory");
}
__device__ __forceinline__ void cl_ld1(unsigned p, double &v)
{
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(p));
}
__device__ __forceinline__ void cl_ld1(unsigned p, float &v)
{
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(p));
}
__device__ __forceinline__ int cl_ldi(unsigned p)
{
    int v;
    asm volatile("ld.shared.s32 %0, [%1];" : "=r"(v) : "r"(p));
    return v;
}
__device__ __forceinline__ void cl_ldu(unsigned p, unsigned long long &a, unsigned long long &b)
{
    asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(p));
}
__device__ __forceinline__ void cl_stu(unsigned p, unsigned long long a, unsigned long long b)
{
    asm volatile("st.shared.v2.u64 [%0], {%1, %2};" ::"r"(p), "l"(a), "l"(b) : "memory");
}

__device__ __forceinline__ void cl_mma(double (&c)[4], double a0, double a1, double a2, double a3, double b0, double b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a0), "d"(a1), "d"(a2), "d"(a3), "d"(b0), "d"(b1));
}

__device__ __forceinline__ unsigned cl_mapa(unsigned p, int rank)
{
    unsigned d;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(p), "r"(rank));
    return d;
}

// 16 bytes to another CTA's shared memory, counted by its mbarrier
__device__ __forceinline__ void cl_send(unsigned dst, unsigned long long a, unsigned long long b, unsigned bar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(dst), "l"(a),
                 "l"(b), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void cl_expect(unsigned bar, int bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// bounded wait for an mbarrier's phase; records the error when it gives up
__device__ __noinline__ bool cl_wait_slow(unsigned bar, unsigned parity, int *status, unsigned long long limit)
{
    const unsigned long long t0 = globaltimer_ns();
    for (;;) {
        for (int spins = 0; spins < 16; spins++) {
            unsigned ok;
            asm volatile(
                "{\n\t.reg .pred P1;\n\t"
                "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P1, [%1], %2;\n\t"
                "selp.b32 %0, 1, 0, P1;\n\t}"
                : "=r"(ok)
                : "r"(bar), "r"(parity)
                : "memory");
            if (ok) return true;
        }
        if (*(volatile int *)&status[1] != 0) return false;
        if (globaltimer_ns() - t0 > limit) {
            record_error(status, ERR_BARRIER_TIMEOUT, 1);
            return false;
        }
    }
}
__device__ __forceinline__ bool cl_wait(unsigned bar, unsigned parity, int *status, unsigned long long limit)
{
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred P1;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P1, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, P1;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok || cl_wait_slow(bar, parity, status, limit);
}

template <typename T, int W>
struct CLeafShared {
    alignas(16) unsigned long long cand[CL_NW][2];  // the warps' candidates: key, position
    alignas(16) unsigned char out[16 + CL_B * sizeof(T)];  // the CTA's candidate of the column
    unsigned long long bar[3];  // messages of even and odd columns; the pivot rows of a block
    int fail;                   // set in a wait, read after the next barrier
    T d[W], inv[W];             // the pivots, their reciprocals
    int piv[W];
    unsigned row[CL_B];         // the block's pivot rows: shared address of column 0 (own slab, or received)
};

// Rows blk + 8 .. of the block's 8 pivot rows, finished; then their products
// off the CTA's rows.  c1 = the position after the block, rem columns right of it.
template <int W, int RT>
__device__ __forceinline__ void cl_update(const CLeafCfg<double, W, RT> *, unsigned slab, unsigned ub, unsigned spos,
                                          const double (&dz)[2], int blk, int rem, int c1)
{
    using C = CLeafCfg<double, W, RT>;
    // a warp's 32 RT rows as 2 RT tiles of 16: fragment row g is tile row pg,
    // so that the rows a quarter-warp touches fall on distinct banks
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int pg = (g >> 1) + ((g & 1) << 2);
    const unsigned r0 = slab + (warp * 32 * RT + pg) * C::PITCH * 8;
    constexpr int MT = RT > 1 && RT % 2 ? 2 : RT > 2 ? 4 : 2 * RT;  // tiles at a time
#pragma unroll 1
    for (int pass = 0; pass < 2 * RT / MT; pass++) {
        const unsigned rp = r0 + pass * MT * 16 * C::PITCH * 8;
        const int row0 = warp * 32 * RT + pass * MT * 16 + pg;
        double a[MT][4];
        unsigned live = 0;
#pragma unroll
        for (int m = 0; m < MT; m++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int row = 16 * m + 8 * h;
                cl_ld1(rp + (row * C::PITCH + blk + t) * 8, a[m][h]);
                cl_ld1(rp + (row * C::PITCH + blk + t + 4) * 8, a[m][2 + h]);
                // -l, and nothing of a zero pivot's column
                a[m][h] = dz[0] == 0.0 ? 0.0 : -a[m][h];
                a[m][2 + h] = dz[1] == 0.0 ? 0.0 : -a[m][2 + h];
                if (cl_ldi(spos + (row0 + row) * 4) >= c1) live |= 1u << (2 * m + h);  // done rows stay
            }
#pragma unroll 1
        for (int n0 = 0; n0 < rem; n0 += 8) {
            double b0, b1;
            cl_ld1(ub + (t * C::UP + n0 + g) * 8, b0);
            cl_ld1(ub + ((t + 4) * C::UP + n0 + g) * 8, b1);
            double lo[MT][2], hi[MT][2];
            const unsigned p = rp + (blk + CL_B + n0 + 2 * t) * 8;
#pragma unroll
            for (int m = 0; m < MT; m++) {
                cl_ld16(p + 16 * m * C::PITCH * 8, lo[m]);
                cl_ld16(p + (16 * m + 8) * C::PITCH * 8, hi[m]);
            }
#pragma unroll
            for (int m = 0; m < MT; m++) {
                // summed from zero, subtracted once: 8 roundings an element
                // over the leaf instead of 64 (forward error of x at n = 2048,
                // 16 systems, geometric mean: 9.1e-13, with this 6.6e-13)
                double c[4] = {0.0, 0.0, 0.0, 0.0};
                cl_mma(c, a[m][0], a[m][1], a[m][2], a[m][3], b0, b1);
                lo[m][0] += c[0];
                lo[m][1] += c[1];
                hi[m][0] += c[2];
                hi[m][1] += c[3];
            }
#pragma unroll
            for (int m = 0; m < MT; m++) {
                if (live >> (2 * m) & 1) cl_st16(p + 16 * m * C::PITCH * 8, lo[m]);
                if (live >> (2 * m + 1) & 1) cl_st16(p + (16 * m + 8) * C::PITCH * 8, hi[m]);
            }
        }
    }
}
template <int W, int RT>
__device__ __forceinline__ void cl_update(const CLeafCfg<float, W, RT> *, unsigned slab, unsigned ub, unsigned spos,
                                          const float (&dz)[8], int blk, int rem, int c1)
{
    using C = CLeafCfg<float, W, RT>;
    // each thread its own rows, two or three at a time
    constexpr int RU = RT % 2 ? 3 : 2;
    static_assert(RT % RU == 0, "whole groups of rows");
    const int tid = threadIdx.x;
#pragma unroll
    for (int k = 0; k < RT; k += RU) {
        float l[RU][CL_B];
        unsigned row[RU];
        bool live[RU];
#pragma unroll
        for (int h = 0; h < RU; h++) {
            const int lr = tid + (k + h) * CL_TPB;
            row[h] = slab + (lr * C::PITCH + blk) * 4;
            live[h] = cl_ldi(spos + lr * 4) >= c1;
#pragma unroll
            for (int j = 0; j < CL_B; j += 4) {
                float v[4];
                cl_ld16(row[h] + j * 4, v);
#pragma unroll
                for (int e = 0; e < 4; e++) l[h][j + e] = dz[j + e] == 0.f ? 0.f : v[e];
            }
        }
#pragma unroll 1
        for (int n0 = 0; n0 < rem; n0 += 4) {
            float c[RU][4];
#pragma unroll
            for (int h = 0; h < RU; h++) cl_ld16(row[h] + (CL_B + n0) * 4, c[h]);
#pragma unroll
            for (int j = 0; j < CL_B; j++) {
                float u[4];
                cl_ld16(ub + (j * C::UP + n0) * 4, u);
#pragma unroll
                for (int h = 0; h < RU; h++)
#pragma unroll
                    for (int e = 0; e < 4; e++) c[h][e] = cl_fnma(l[h][j], u[e], c[h][e]);
            }
#pragma unroll
            for (int h = 0; h < RU; h++)
                if (live[h]) cl_st16(row[h] + (CL_B + n0) * 4, c[h]);
        }
    }
}

// REF: one of the reference's pivot rules, whose searches look at multipliers
// (64 columns by plain partial pivoting without them in the chain: 200 rows
// 56 -> 52 us, 4096 rows 79.5 -> 77)
template <typename T, int W, int RT, bool REF>
__global__ void __launch_bounds__(CL_ALL, 1) cluster_leaf_kernel(const CLeafParams<T> P)
{
    using C = CLeafCfg<T, W, RT>;
    constexpr int VEC = C::VEC, PITCH = C::PITCH, MSG = C::MSG, PIECES = C::PIECES;
    constexpr unsigned ES = sizeof(T);
    extern __shared__ __align__(16) unsigned char cl_dyn[];
    __shared__ CLeafShared<T, W> sh;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int CL = gridDim.x, rank = blockIdx.x;  // one cluster per launch
    const int c0 = P.c0, w = P.w;
    const int rb = c0 + rank * P.rpc, nr = max(0, min(P.rpc, P.n - rb));
    const unsigned slab = cl_smem(cl_dyn + C::O_SLAB), ub = cl_smem(cl_dyn + C::O_U), xb = cl_smem(cl_dyn + C::O_X);
    const unsigned msg = cl_smem(cl_dyn + C::O_MSG), spos = cl_smem(cl_dyn + C::O_POS), out = cl_smem(sh.out);
    const unsigned cands = cl_smem(&sh.cand[0][0]), bar0 = cl_smem(&sh.bar[0]), failed = cl_smem(&sh.fail);

    // the CTA's rows, 16 bytes per copy (zeros past column w)
    constexpr int CPR = W / VEC;  // copies per row
    for (int q = tid; q < nr * CPR; q += CL_ALL) {
        const int lr = q / CPR, ch = q % CPR;
        const int have = min(VEC, max(0, w - ch * VEC)) * (int)ES;
        const T *src = P.a + (size_t)(rb + lr) * P.ld + c0 + (have ? ch * VEC : 0);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(slab + (lr * PITCH + ch * VEC) * ES), "l"(src),
                     "r"(have)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (tid == 0) {
        sh.fail = *(volatile int *)&P.status[1] != 0;  // an earlier wait of this call gave up: nothing to do
        for (int b = 0; b < 3; b++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8 * b) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // the barriers exist before any CTA sends to them
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    __syncthreads();

    // row k of this thread: tid + k CL_TPB of the CTA's (helpers have none)
    const bool help = tid >= CL_TPB;
    T r[RT][CL_B];  // its columns of the block from the current one on
    T ls[RT];       // the multiplier the reference's pivot searches look at
    int pos[RT];    // its current position (rows of the view); -1: no row
#pragma unroll
    for (int k = 0; k < RT; k++) {
        pos[k] = !help && tid + k * CL_TPB < nr ? rb + tid + k * CL_TPB : -1;
        ls[k] = T(0);
    }
    const unsigned slot = slab + tid * PITCH * ES;  // of this thread's first row
    // this thread's sends of a column's message: piece tid % 8 to CTA tid / 8
    const int to = tid >> 3, piece = tid & 7;
    const bool sends = CL > 1 && to < CL && piece < PIECES && rank != P.withhold;
    const unsigned rmsg = cl_mapa(msg + rank * MSG + piece * 16, sends ? to : 0), rbar = cl_mapa(bar0, sends ? to : 0);
    // a helper's sends of a pivot row: 16-byte piece lane, to CTAs hw, hw + 4, ...
    const int hw = warp - CL_NW;
    const int mode = P.mode, goff = P.goff;

    bool ok = sh.fail == 0;
#pragma unroll 1
    for (int blk = 0; ok && blk < w; blk += CL_B) {
        const int nbk = min(CL_B, w - blk), rem = w - blk - CL_B;
        const int rowp = rem > 0 && CL > 1 ? (w - blk + VEC - 1) / VEC : 0;  // 16-byte pieces of a pivot row sent on
        if (rowp && tid == 0) cl_expect(bar0 + 16, nbk * rowp * 16);
        if (!help)
#pragma unroll
            for (int k = 0; k < RT; k++)
#pragma unroll
                for (int j = 0; j < CL_B; j += VEC) {
                    T v[VEC];
                    cl_ld16(slot + (k * CL_TPB * PITCH + blk + j) * ES, v);
#pragma unroll
                    for (int e = 0; e < VEC; e++) r[k][j + e] = v[e];
                }
#pragma unroll 1
        for (int jb = 0; jb < nbk; jb++) {
            const int ip = blk + jb, c = c0 + ip, par = ip & 1;
            if (!help) {
                // lu2tlib.c:1052, counted over the whole matrix; as in leaf_kernel the first
                // column of each 16 searches itself (odd when a slab begins at an odd row)
                const bool use_ls = REF && (ip & 15) && (mode == PIVOT_REF_FIRST || ((c + goff) & 1));
                // this thread's candidate, the warp's, the CTA's
                unsigned long long key = 0;
                int kp = INT_MAX, kr = 0;
                T kd = T(1);
#pragma unroll
                for (int k = 0; k < RT; k++) {
                    T v = r[k][0];
                    if (use_ls) v = ls[k];
                    const int pk = pos[k];
                    const unsigned long long kk = cl_key(v, pk >= c, pk == c);
                    const bool take = (kk > key) | ((kk == key) & (pk < kp) & (kk != 0));
                    key = take ? kk : key;
                    kp = take ? pk : kp;
                    kr = take ? k : kr;
                    kd = take ? r[k][0] : kd;
                }
                // the columns after this one scaled, the pivot last: of use to
                // one lane of the CTA, but made beside the search, not after it
                T x[CL_B];
                const T inv = cl_zero(kd) ? T(1) : T(1) / kd;
#pragma unroll
                for (int j = 0; j < CL_B; j++) {
                    x[j] = r[0][(j + 1) % CL_B];
#pragma unroll
                    for (int k = 1; k < RT; k++) x[j] = kr == k ? r[k][(j + 1) % CL_B] : x[j];
                    if (j + 1 < CL_B) x[j] *= inv;
                }
                const int wl = cl_winner(key, kp, lane);
                if (lane == wl) cl_stu(cands + 16 * warp, key, (unsigned)kp);
                __syncthreads();
                unsigned long long ck = 0ull, cp = INT_MAX;
                if (lane < CL_NW) cl_ldu(cands + 16 * lane, ck, cp);
                if (cl_ldi(failed)) {
                    ok = false;
                    break;
                }
                if (warp == cl_winner(ck, (int)(unsigned)cp, lane) && lane == wl) {
                    cl_stu(out, key, (unsigned)kp | (unsigned long long)(unsigned)(tid + kr * CL_TPB) << 32);
#pragma unroll
                    for (int j = 0; j < CL_B; j += VEC) {
                        T v[VEC];
#pragma unroll
                        for (int e = 0; e < VEC; e++) v[e] = x[j + e];
                        cl_st16(out + 16 + j * ES, v);
                    }
                }
            } else {
                __syncthreads();
                if (cl_ldi(failed)) {
                    ok = false;
                    break;
                }
            }
            __syncthreads();
            unsigned bst = out;
            int wc = 0;
            bool got = true;
            if (CL > 1) {
                const unsigned bar = bar0 + 8 * par;
                if (tid == 0) cl_expect(bar, CL * MSG);
                if (sends) {
                    unsigned long long v0, v1;
                    cl_ldu(out + piece * 16, v0, v1);
                    cl_send(rmsg + par * CL_MAXC * MSG, v0, v1, rbar + 8 * par);
                }
                // every CTA's candidate of this column (after a failed wait what
                // is read below is nobody's row, and the CTA leaves at its next
                // barrier: its mbarriers may not be armed again)
                got = cl_wait(bar, (unsigned)(ip >> 1) & 1u, P.status, P.wait_ns);
                if (!got) sh.fail = 1;
                __syncwarp();
                const unsigned m0 = msg + par * CL_MAXC * MSG;
                unsigned long long ck = 0ull, cp = INT_MAX;
                if (lane < CL) cl_ldu(m0 + lane * MSG, ck, cp);
                wc = cl_winner(ck, (int)(unsigned)cp, lane);
                bst = m0 + wc * MSG;
            }
            const int p = cl_ldi(bst + 8);
            if (!help) {
                T u[CL_B];
#pragma unroll
                for (int j = 0; j < CL_B; j += VEC) {
                    T v[VEC];
                    cl_ld16(bst + 16 + j * ES, v);
#pragma unroll
                    for (int e = 0; e < VEC; e++) u[j + e] = v[e];
                }
                const bool zero = cl_zero(u[CL_B - 1]);
#pragma unroll
                for (int k = 0; k < RT; k++) {
                    const T l = r[k][0];
                    const int pk = pos[k];
                    // rows that are done compute values nobody reads
                    if (!zero) {
#pragma unroll
                        for (int j = 0; j + 1 < CL_B; j++) r[k][j] = cl_fnma(l, u[j], r[k][j + 1]);
                    } else {
#pragma unroll
                        for (int j = 0; j + 1 < CL_B; j++) r[k][j] = r[k][j + 1];
                    }
                    if ((pk >= c) & (pk != p)) cl_st1(slot + (k * CL_TPB * PITCH + ip) * ES, l);
                    pos[k] = pk == p ? c : (pk == c ? p : pk);
                    if (REF && (mode == PIVOT_REF || ip == 0)) ls[k] = l;
                }
            } else {
                if (rowp) {
                    // the rest of the pivot row, as it was before the block, and its
                    // multipliers so far: to all CTAs from its own
                    if (rank == wc && got && lane < rowp && rank != P.withhold) {
                        const unsigned row = slab + ((unsigned)cl_ldi(bst + 12) * PITCH + blk) * ES + lane * 16;
                        unsigned long long v0, v1;
                        cl_ldu(row, v0, v1);
#pragma unroll 1
                        for (int dst = hw; dst < CL; dst += CL_HELP / 32)
                            cl_send(cl_mapa(xb + (jb * C::XP + blk) * ES + lane * 16, dst), v0, v1,
                                    cl_mapa(bar0 + 16, dst));
                    }
                } else if (hw == 1 && lane == 0) {
                    sh.row[jb] = CL > 1 ? 0u : slab + (unsigned)cl_ldi(bst + 12) * PITCH * ES;
                }
                // row c of the factors, the block's columns from c on
                if (hw == 0 && lane < CL_B) {
                    T v;
                    cl_ld1(bst + 16 + ((lane + CL_B - 1) & (CL_B - 1)) * ES, v);  // the pivot, then the columns after it
                    if (rank == 0 && lane < nbk - jb) P.a[(size_t)c * P.ld + c + lane] = v;
                    if (lane == 0) {
                        sh.d[ip] = v;
                        sh.piv[ip] = p;
                    }
                }
            }
        }
        if (!ok) break;
        if (!help)
#pragma unroll
            for (int k = 0; k < RT; k++)
                asm volatile("st.shared.s32 [%0], %1;" ::"r"(spos + (tid + k * CL_TPB) * 4), "r"(pos[k]) : "memory");
        if (rowp && tid < CL_B) sh.row[tid] = xb + tid * C::XP * ES;
        if (rowp && !cl_wait(bar0 + 16, (unsigned)(blk / CL_B) & 1u, P.status, P.wait_ns)) sh.fail = 1;
        __syncthreads();
        if (sh.fail) break;
        if (rem <= 0) break;  // the last block
        // the 8 pivot rows right of the block, one column per thread (zeros past w), in
        // whole warps: lanes 0..7 hold the reciprocals.  (The shuffle tells the compiler
        // that a warp takes the branch as one: n = 3333 5875 -> 5795 us.)
        if (__shfl_sync(0xffffffffu, warp, 0) * 32 < rem) {
            const int col = blk + CL_B + tid;
            const T dl = sh.d[blk + (lane & (CL_B - 1))], il = cl_zero(dl) ? T(1) : T(1) / dl;
            T x[CL_B], lij[CL_B][CL_B];
#pragma unroll
            for (int j = 0; j < CL_B; j++) {
                const unsigned row = (unsigned)cl_ldi(cl_smem(&sh.row[j]));
                x[j] = T(0);
                if (tid < rem) cl_ld1(row + col * ES, x[j]);
#pragma unroll
                for (int i = 0; i < j; i += VEC) {
                    T v[VEC];
                    cl_ld16(row + (blk + i) * ES, v);
#pragma unroll
                    for (int e = 0; e < VEC; e++) lij[j][i + e] = v[e];
                }
            }
#pragma unroll
            for (int j = 0; j < CL_B; j++) {
                T v = x[j];
#pragma unroll
                for (int i = 0; i < j; i++) v = cl_fnma(lij[j][i], x[i], v);
                v *= __shfl_sync(0xffffffffu, il, j);
                if (rank == 0 && tid < rem) P.a[(size_t)(c0 + blk + j) * P.ld + c0 + col] = v;
                x[j] = cl_zero(__shfl_sync(0xffffffffu, dl, j)) ? T(0) : v;  // a zero pivot's column subtracts nothing
                if (W > 16 || tid < 8) cl_st1(ub + (j * C::UP + tid) * ES, x[j]);  // (16 columns: at most 8 of them)
            }
        }
        __syncthreads();
        if (!help) {
            if constexpr (sizeof(T) == 8) {
                const T dz[2] = {sh.d[blk + (lane & 3)], sh.d[blk + (lane & 3) + 4]};
                cl_update(static_cast<const C *>(nullptr), slab, ub, spos, dz, blk, rem, c0 + blk + CL_B);
            } else {
                T dz[CL_B];
#pragma unroll
                for (int j = 0; j < CL_B; j++) dz[j] = sh.d[blk + j];
                cl_update(static_cast<const C *>(nullptr), slab, ub, spos, dz, blk, rem, c0 + blk + CL_B);
            }
        }
        __syncthreads();
    }
    __syncthreads();
    if (!sh.fail) {
        // the pivots, their reciprocals, then the multipliers to the rows' last
        // positions; a pivot row's are scaled by its 1/pivot like the rest of
        // it, and its columns from its own on are in the matrix already
        if (tid < w) {
            const T d = sh.d[tid], inv = cl_zero(d) ? T(1) : T(1) / d;
            sh.inv[tid] = inv;
            if (rank == 0) {
                P.ipiv[c0 + tid] = sh.piv[tid] + P.goff;
                P.dinv[c0 + tid] = inv;
                if (cl_zero(d)) atomicMin(&P.status[0], c0 + tid + 1);
            }
        }
        __syncthreads();
        for (int q = tid; q < nr * CPR; q += CL_ALL) {
            const int lr = q / CPR, ch = q % CPR;
            const int at = cl_ldi(spos + lr * 4), have = min(w, at - c0) - ch * VEC;
            if (have <= 0) continue;
            T *dst = P.a + (size_t)at * P.ld + c0 + ch * VEC;
            T v[VEC];
            cl_ld16(slab + (lr * PITCH + ch * VEC) * ES, v);
            if (at < c0 + w) {
#pragma unroll
                for (int e = 0; e < VEC; e++) v[e] *= sh.inv[at - c0];
            }
            if (have >= VEC) {
                cl_put16(dst, v);
            } else {
#pragma unroll
                for (int e = 0; e < VEC; e++)
                    if (e < have) dst[e] = v[e];
            }
        }
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    // a CTA that gave up has not waited for all that was sent to it, and the barrier
    // does not order st.async: its shared memory stays until the last of it has landed
    // (all was sent before the barrier; 16 CTAs' messages take 0.6 us)
    if (CL > 1 && sh.fail) {
        const unsigned long long t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < CL_LINGER_NS) {
        }
    }
}

// ---------------------------------------------------------------------------
// The widest slab whose rows one cluster of 16 holds, by rows (each CTA
// 128-170 KB of shared memory, the tall instances 210-226 KB):
//   FP64: 64 columns to 4096 rows, 32 to 8192, tall 12288, 16 to 16384, tall 20480
//   FP32: 64 columns to 8192 rows, tall 12288, 32 to 16384, tall 24576, 16 to 32768
// A wider leaf replaces whole levels of the panel recursion (four launches
// each).  The tall instances fill the SM's shared memory (FP32, 12288 rows: 64
// columns 90 us against twice 51 and those launches; FP64: 32 columns 57
// against twice 34; 16 columns of about 20000 rows beside an update 33 us,
// over the whole grid 151).  Taller panels go to leaf_kernel.
template <typename T, int W, bool TALL>
using CLeafPick = CLeafCfg<T, W, sizeof(T) == 8 ? (TALL ? 64 / W + 1 : 64 / W) : (TALL ? 192 / W : 128 / W)>;

template <typename T, int W, bool TALL>
static constexpr int cl_rows()
{
    return CL_MAXC * CLeafPick<T, W, TALL>::ROWS;
}

// shared memory and cluster size limits of one instance, in the current context
template <typename T, int W, bool TALL, bool REF>
static cudaError_t cl_attributes()
{
    using C = CLeafPick<T, W, TALL>;
    auto kern = cluster_leaf_kernel<T, W, C::ROWS / CL_TPB, REF>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}

// true when a cluster of 16 of this instance can be resident
template <typename T, int W, bool TALL, bool REF>
static bool cl_prepare_1()
{
    using C = CLeafPick<T, W, TALL>;
    auto kern = cluster_leaf_kernel<T, W, C::ROWS / CL_TPB, REF>;
    if (cl_attributes<T, W, TALL, REF>() != cudaSuccess) return false;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(CL_ALL);
    cfg.dynamicSmemBytes = C::SMEM;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {16, 1, 1};
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int clusters = 0;
    return cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) == cudaSuccess && clusters >= 1;
}

template <typename T, int W, bool TALL = false>
static bool cl_prepare(bool query)
{
    if (query) return cl_prepare_1<T, W, TALL, false>() && cl_prepare_1<T, W, TALL, true>();
    return cl_attributes<T, W, TALL, false>() == cudaSuccess && cl_attributes<T, W, TALL, true>() == cudaSuccess;
}

// whether a device takes the cluster leaf: 0 not asked yet, else 1 or -1
static std::atomic<signed char> cl_known[128];

// The instances' sizes belong to the CUDA context and are gone after
// cudaDeviceReset: set whenever a library context is made (for every launch they
// cost the precision forms 0.5 us a leaf), the FP64 instances of up to 4096 rows
// also by the allocation-free solve, which has none.
bool cluster_leaf_setup(bool small)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 128) return false;
    const signed char known = cl_known[dev].load();
    if (known < 0) return false;
    const bool query = known == 0;
    bool ok = cl_prepare<double, 64>(query) && cl_prepare<double, 32>(query) && cl_prepare<double, 16>(query);
    if (!small || query)
        ok = ok && cl_prepare<float, 64>(query) && cl_prepare<float, 32>(query) && cl_prepare<float, 16>(query) &&
             cl_prepare<double, 32, true>(query) && cl_prepare<double, 16, true>(query) &&
             cl_prepare<float, 64, true>(query) && cl_prepare<float, 32, true>(query);
    if (query) cl_known[dev].store(ok ? 1 : -1);
    cudaGetLastError();
    return ok;
}

static bool cl_device_ok()
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 128) return false;
    const signed char known = cl_known[dev].load();
    return known ? known > 0 : cluster_leaf_setup(false);
}

// columns the leaf takes for `rows` rows, in the tall instance or not; 0: not this leaf
template <typename T>
static int cl_width(int rows, int max_ctas, bool &tall)
{
    tall = false;
    if (rows <= 0 || max_ctas < 16 || !cl_device_ok()) return 0;
    if (rows <= cl_rows<T, 64, false>()) return 64;
    tall = sizeof(T) == 4 && rows <= cl_rows<float, 64, true>();
    if (tall) return 64;
    if (rows <= cl_rows<T, 32, false>()) return 32;
    tall = rows <= cl_rows<T, 32, true>();
    if (tall) return 32;
    if (rows <= cl_rows<T, 16, false>()) return 16;
    tall = sizeof(T) == 8 && rows <= cl_rows<double, 16, true>();
    return tall ? 16 : 0;
}

int leaf_width(int rows, size_t tsize, int max_ctas)
{
    bool tall;
    const int k = tsize == sizeof(double) ? cl_width<double>(rows, max_ctas, tall) : cl_width<float>(rows, max_ctas, tall);
    return k > 16 ? k : 16;
}

template <typename T, int W, bool TALL, bool REF>
static cudaError_t cl_launch_1(CLeafParams<T> P, cudaStream_t st)
{
    using C = CLeafPick<T, W, TALL>;
    const int rows = P.n - P.c0;
    int cl = 1;
    while (cl < 16 && cl * C::ROWS < rows) cl *= 2;
    P.rpc = (rows + cl - 1) / cl;
    if (P.rpc > C::ROWS) return cudaErrorInvalidConfiguration;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)cl);
    cfg.blockDim = dim3(CL_ALL);
    cfg.dynamicSmemBytes = C::SMEM;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {(unsigned)cl, 1, 1};
    cfg.attrs = at;
    cfg.numAttrs = 1;
    count_launch();
    return cudaLaunchKernelEx(&cfg, cluster_leaf_kernel<T, W, C::ROWS / CL_TPB, REF>, P);
}

template <typename T, int W, bool TALL = false>
static cudaError_t cl_launch_w(const CLeafParams<T> &P, cudaStream_t st)
{
    return P.mode == PIVOT_PARTIAL ? cl_launch_1<T, W, TALL, false>(P, st) : cl_launch_1<T, W, TALL, true>(P, st);
}

template <typename T>
static cudaError_t launch_leaf_cluster_t(T *a, long ld, int n, int c0, int w, int mode, int goff, int *ipiv, T *dinv,
                                         const LeafBuffers &buf, int *status, int max_ctas, cudaStream_t st,
                                         bool *used)
{
    *used = false;
    bool tall;
    const int width = cl_width<T>(n - c0, max_ctas, tall);
    constexpr int VEC = 16 / (int)sizeof(T);
    // 16-byte copies of row segments
    if (w <= 0 || w > width || (reinterpret_cast<uintptr_t>(a) & 15) || ld % VEC || c0 % VEC) return cudaSuccess;
    *used = true;
    const CLeafParams<T> P{a, ld, n, c0, w, 0, mode, goff, ipiv, dinv, status, buf.wait_ns, buf.withhold};
    // a narrower slab has more rows in its base instance than a wider tall one
    if (w <= 16 && n - c0 <= cl_rows<T, 16, false>()) return cl_launch_w<T, 16>(P, st);
    if (w <= 32 && n - c0 <= cl_rows<T, 32, false>()) return cl_launch_w<T, 32>(P, st);
    if (!tall) return cl_launch_w<T, 64>(P, st);
    if constexpr (sizeof(T) == 8)
        return width == 16 ? cl_launch_w<T, 16, true>(P, st) : cl_launch_w<T, 32, true>(P, st);
    else
        return width == 32 ? cl_launch_w<T, 32, true>(P, st) : cl_launch_w<T, 64, true>(P, st);
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

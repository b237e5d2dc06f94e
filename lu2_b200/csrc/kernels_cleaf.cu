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
// that no amount of bandwidth shortens, and the instructions that every warp
// of a CTA spends on it.  Over the whole grid that chain costs four trips
// through L2 per column (kernels_leaf.cu: 3.6-4.6 us); inside a cluster it is
// two CTA barriers and one trip through distributed shared memory.  So:
//  * S neighbouring lanes hold R whole rows in registers, a row's columns dealt
//    to them in turn; lane q of the S also keeps the book of rows q, q + S, ...
//    of the R (their position, their part in the pivot search).  One lane per
//    row would read the pivot row from shared memory R times as often, one
//    book per lane and row would repeat its work S times.  256 threads, since
//    whatever all warps do costs issue slots per warp.
//  * no row ever moves: an exchange c <-> p is two rows changing their
//    positions (`pos`), and a row is written back to its last one at the end.
//  * the registers rotate: after S columns the rows move down by one register,
//    so the columns are one rolled loop (its current column always in register
//    0), small enough for the instruction cache (a body unrolled over the S
//    columns and four widths measured 1.75 us a column, most of it fetch).
//    The multiplier l goes to the row's shared-memory slot, which is stored to
//    the matrix at the end.
//  * a warp's candidate is found with redux.sync on the bits of |a| (the upper
//    word decides except in ties), the CTA's from the warps' after one
//    barrier; its owner puts the row, already scaled by 1/pivot, into shared
//    memory, from where after a second barrier all warps send it to every CTA
//    of the cluster with st.async, which completes an mbarrier there.  Every
//    warp then picks the winner from the CTAs' candidates by itself.  (Sending
//    the candidates' keys first and the winner's row alone in a second trip
//    measured 1000-1300 cycles a column against 750-1100 for the one trip.)
// Messages are double-buffered by column parity: a CTA can be one column ahead
// of another at most, since it needs that CTA's message of a column to leave
// it, and a buffer's readers have passed the next column's CTA barriers before
// their CTA sends that column's message.
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

template <typename T, int W, int S, int R, int TPB>
struct CLeafCfg {
    static constexpr int NW = TPB / 32;
    static constexpr int VEC = 16 / (int)sizeof(T);
    static constexpr int PITCH = W + VEC;     // a slot's 16-byte accesses by consecutive rows hit distinct banks
    static constexpr int ROWS = R * TPB / S;  // rows a CTA holds
    static constexpr int ROWB = (W + S * VEC) * (int)sizeof(T);  // a travelling row: each lane's part and 16 bytes of padding
    static constexpr int MSG = 16 + ROWB;                        // header (key, position), then the row
    static constexpr int MAXC = 16;
    static constexpr size_t O_SLAB = 0;
    static constexpr size_t O_MSG = O_SLAB + (size_t)ROWS * PITCH * sizeof(T);
    static constexpr size_t O_POS = O_MSG + (size_t)2 * MAXC * MSG;
    static constexpr size_t SMEM = O_POS + (size_t)ROWS * sizeof(int);
};

__device__ __forceinline__ unsigned cl_smem(const void *p)
{
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

// Pivot candidates order as (key, then lower position): key 0 = not a
// candidate, 1 = row c when nothing else is left (a column of NaNs keeps its
// row), else the bits of |v| + 2 -- for float in the upper word.  A thread's
// best of its rows is kept as a value: -2 for none, -1 for such a row c.
__device__ __forceinline__ unsigned long long cl_key(double best)
{
    return best >= 0.0 ? (unsigned long long)__double_as_longlong(best) + 2ull : (best > -1.5 ? 1ull : 0ull);
}
__device__ __forceinline__ unsigned long long cl_key(float best)
{
    return (unsigned long long)(best >= 0.f ? __float_as_uint(best) + 2u : (best > -1.5f ? 1u : 0u)) << 32;
}
__device__ __forceinline__ bool cl_zero(double v) { return ((unsigned long long)__double_as_longlong(v) << 1) == 0; }
__device__ __forceinline__ bool cl_zero(float v) { return (__float_as_uint(v) << 1) == 0; }

// the lane holding the warp's best candidate
__device__ __forceinline__ int cl_winner(unsigned long long key, int pos, int lane)
{
    const unsigned full = 0xffffffffu, hi = (unsigned)(key >> 32), lo = (unsigned)key;
    const unsigned mh = __reduce_max_sync(full, hi);
    bool in = hi == mh;
    const unsigned b = __ballot_sync(full, in);
    unsigned win = __reduce_min_sync(full, in ? (unsigned)lane : 31u);
    if (b & (b - 1)) {  // a tie in the upper word
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

// One CTA's part in the columns of the leaf
template <typename T, int W, int S, int R, int TPB>
struct CLeaf {
    using C = CLeafCfg<T, W, S, R, TPB>;
    static constexpr int NW = C::NW, VEC = C::VEC, PITCH = C::PITCH, MSG = C::MSG;
    static constexpr int WL = W / S;         // columns of a row per lane
    static constexpr int M = R / S;          // rows a lane keeps the book of
    static constexpr int LSTR = WL + VEC;    // elements between the lanes' parts of a travelling row
    static constexpr int PPL = WL / VEC;     // 16-byte pieces per lane's part
    static_assert(R % S == 0 && W % S == 0 && WL % VEC == 0, "rows and columns dealt evenly");
    struct Shared {
        alignas(16) unsigned long long cand[NW][2];  // the warps' candidates: key, position
        int fail;             // set in a column's wait, read after the next column's first barrier
        unsigned long long bar[2];
        T d[W], inv[W];  // the pivots, at the end their reciprocals
        int piv[W];
        alignas(16) unsigned char out[MSG];       // the CTA's candidate of the column
        alignas(16) unsigned char none[C::ROWB];  // zeros: what a zero pivot's column subtracts
    };
    struct Rows {
        T r[R][WL];  // row k, register i of lane q: column i S + q of what is left
        T ls[M];     // row m S + q: the multiplier the reference's pivot searches look at
        int pos[M];  // its current position (rows of the view); -1: no row
    };

    // Every column of the leaf; false when a wait gave up.
    static __device__ __forceinline__ bool columns(const CLeafParams<T> &P, Shared &sh, unsigned char *dyn, Rows &x)
    {
        const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = lane % S;
        const int CL = gridDim.x, rank = blockIdx.x, w = P.w;
        constexpr unsigned ES = sizeof(T);
        const unsigned slot = cl_smem(dyn + C::O_SLAB) + tid * PITCH * ES;  // of this lane's first row
        const unsigned msg = cl_smem(dyn + C::O_MSG), out = cl_smem(sh.out), none = cl_smem(sh.none);
        const unsigned cands = cl_smem(&sh.cand[0][0]), failed = cl_smem(&sh.fail);
        // this thread's share of the sends: pieces p0, p0 + tpd, ... to CTA `to`
        const int tpd = TPB / CL, to = tid / tpd, p0 = tid - to * tpd;
        const unsigned bar0 = cl_smem(&sh.bar[0]);
        unsigned rmsg, rbar;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rmsg) : "r"(msg + rank * MSG), "r"(to));
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rbar) : "r"(bar0), "r"(to));

#pragma unroll 1
        for (int ip = 0; ip < w; ip++) {
            const int c = P.c0 + ip, par = ip & 1, s = ip % S, left = w - ip + s;  // columns from the group's first on
            const bool use_ls = ip > 0 && ((P.mode == PIVOT_REF && ((c + P.goff) & 1)) ||  // lu2tlib.c:1052
                                           P.mode == PIVOT_REF_FIRST);
            // the column to all lanes of its rows (they are the multipliers)
            T l[R], lm[M];
#pragma unroll
            for (int k = 0; k < R; k++) l[k] = S == 1 ? x.r[k][0] : __shfl_sync(0xffffffffu, x.r[k][0], lane - q + s);
            // this thread's candidate, the warp's, the CTA's
            T best = T(-2), kd = T(1);
            int kp = INT_MAX, kr = 0;
#pragma unroll
            for (int m = 0; m < M; m++) {
                lm[m] = l[m * S];
#pragma unroll
                for (int e = 1; e < S; e++) lm[m] = q == e ? l[m * S + e] : lm[m];
                T v = lm[m];
                if (use_ls) v = x.ls[m];
                v = fabs(v);
                const int pm = x.pos[m];
                const bool act = pm >= c;
                bool take = act & ((v > best) | ((v == best) & (pm < kp)));
                const bool keep = act & (pm == c) & (best < T(-1)) & !take;
                best = take ? v : (keep ? T(-1) : best);
                take |= keep;
                kp = take ? pm : kp;
                kr = take ? m * S + q : kr;
                kd = take ? lm[m] : kd;
            }
            const unsigned long long key = cl_key(best);
            const int wl = cl_winner(key, kp, lane);
            if (lane == wl) cl_stu(cands + 16 * warp, key, (unsigned)kp);
            __syncthreads();
            unsigned long long ck = 0ull, cp = INT_MAX;
            if (lane < NW) cl_ldu(cands + 16 * lane, ck, cp);
            if (cl_ldi(failed)) return false;
            if (warp == cl_winner(ck, (int)cp, lane)) {
                T inv = cl_zero(kd) ? T(1) : T(1) / kd;
                inv = __shfl_sync(0xffffffffu, inv, wl);
                kr = __shfl_sync(0xffffffffu, kr, wl);
                if (lane / S == wl / S) {
                    const unsigned dst = out + 16 + q * LSTR * ES;
#pragma unroll
                    for (int k = 0; k < R; k++)
                        if (kr == k) {
#pragma unroll
                            for (int j = 0; j < WL; j += VEC)
                                if (j * S < left) {
                                    T v[VEC];
#pragma unroll
                                    for (int e = 0; e < VEC; e++)
                                        v[e] = j + e == 0 && q == s ? x.r[k][0] : x.r[k][j + e] * inv;
                                    cl_st16(dst + j * ES, v);
                                }
                        }
                }
                if (lane == wl) cl_stu(out, key, (unsigned)kp);
            }
            __syncthreads();
            unsigned bst = out;
            if (CL > 1) {
                const int pieces = 1 + S * min(PPL, (left - 1) / (S * VEC) + 1);
                if (tid == 0)
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar0 + 8 * par),
                                 "r"(CL * 16 * pieces)
                                 : "memory");
                if (rank != P.withhold)
#pragma unroll 1
                    for (int i = p0; i < pieces; i += tpd) {
                        // header, then register pieces by lane
                        const unsigned at = i == 0 ? 0 : 16 + ((i - 1) % S) * LSTR * ES + ((i - 1) / S) * 16;
                        unsigned long long v0, v1;
                        cl_ldu(out + at, v0, v1);
                        asm volatile(
                            "st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(
                                rmsg + par * C::MAXC * MSG + at),
                            "l"(v0), "l"(v1), "r"(rbar + 8 * par)
                            : "memory");
                    }
                // every CTA's candidate of this column
                if (!arrived(P, bar0 + 8 * par, (unsigned)(ip >> 1) & 1u)) sh.fail = 1;  // leaves at the next barrier
                __syncwarp();
                const unsigned m0 = msg + par * C::MAXC * MSG;
                ck = 0ull;
                cp = INT_MAX;
                if (lane < CL) cl_ldu(m0 + lane * MSG, ck, cp);
                bst = m0 + cl_winner(ck, (int)cp, lane) * MSG;
            }
            const int p = cl_ldi(bst + 8);
            const unsigned u = bst + 16;
            T d;
            cl_ld1(u + s * LSTR * ES, d);
            unsigned uq = u + q * LSTR * ES;
            if (cl_zero(d)) {
                uq = none;
#pragma unroll
                for (int k = 0; k < R; k++) l[k] = T(0);
            }
            // the pivot row's part of this lane
            T v[WL];
#pragma unroll
            for (int j = 0; j < WL; j += VEC)
                if (j * S < left) {
                    T t[VEC];
                    cl_ld16(uq + j * ES, t);
#pragma unroll
                    for (int e = 0; e < VEC; e++) v[j + e] = t[e];
                }
#pragma unroll
            for (int m = 0; m < M; m++) {
                const int pm = x.pos[m];
                if (pm >= c && pm != p) cl_st1(slot + (m * TPB * PITCH + ip) * ES, lm[m]);
                x.pos[m] = pm == p ? c : (pm == c ? p : pm);
                if (P.mode == PIVOT_REF || ip == 0) x.ls[m] = lm[m];
            }
            // rank-1 update; rows that are done compute values nobody reads, as
            // do lanes up to s in register 0.  After the last of S columns the
            // rows move down by a register.
            if (s != S - 1) {
#pragma unroll
                for (int j = 0; j < WL; j += VEC)
                    if (j * S < left) {
#pragma unroll
                        for (int e = 0; e < VEC; e++)
#pragma unroll
                            for (int k = 0; k < R; k++) x.r[k][j + e] = cl_fnma(l[k], v[j + e], x.r[k][j + e]);
                    }
            } else {
#pragma unroll
                for (int j = 0; j < WL; j += VEC)
                    if (j * S < left) {
#pragma unroll
                        for (int e = 0; e < VEC; e++)
                            if (j + e > 0) {
#pragma unroll
                                for (int k = 0; k < R; k++) x.r[k][j + e - 1] = cl_fnma(l[k], v[j + e], x.r[k][j + e]);
                            }
                    }
            }
            // row c of the factors from column c on (the warps take turns)
            if (warp == (ip & (NW - 1))) {
                if (rank == 0) {
                    T *dst = P.a + (size_t)c * P.ld + c - s;  // column c - s + j: part j % S, register j / S
                    for (int j = s + lane; j < left; j += 32) {
                        T t;
                        cl_ld1(u + ((j % S) * LSTR + j / S) * ES, t);
                        dst[j] = t;
                    }
                }
                if (lane == 0) {
                    sh.d[ip] = d;
                    sh.piv[ip] = p;
                }
            }
        }
        return true;
    }

    // bounded wait for a column's messages; records the error when it gives up
    static __device__ __forceinline__ bool arrived(const CLeafParams<T> &P, unsigned bar, unsigned parity)
    {
        unsigned long long t0 = 0;
#pragma unroll 1
        for (unsigned spins = 1;; spins++) {
            unsigned ok;
            asm volatile(
                "{\n\t.reg .pred P1;\n\t"
                "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P1, [%1], %2;\n\t"
                "selp.b32 %0, 1, 0, P1;\n\t}"
                : "=r"(ok)
                : "r"(bar), "r"(parity)
                : "memory");
            if (ok) return true;
            if ((spins & 15u) == 0) {
                const unsigned long long now = globaltimer_ns();
                if (t0 == 0) t0 = now;
                if (*(volatile int *)&P.status[1] != 0) return false;
                if (now - t0 > P.wait_ns) {
                    record_error(P.status, ERR_BARRIER_TIMEOUT, 1);
                    return false;
                }
            }
        }
    }
};

template <typename T, int W, int S, int R, int TPB>
__global__ void __launch_bounds__(TPB, 1) cluster_leaf_kernel(const CLeafParams<T> P)
{
    using C = CLeafCfg<T, W, S, R, TPB>;
    using L = CLeaf<T, W, S, R, TPB>;
    constexpr int VEC = C::VEC, PITCH = C::PITCH;
    extern __shared__ __align__(16) unsigned char cl_dyn[];
    __shared__ typename L::Shared sh;
    T *slab = reinterpret_cast<T *>(cl_dyn + C::O_SLAB);
    int *spos = reinterpret_cast<int *>(cl_dyn + C::O_POS);
    const int tid = threadIdx.x, rank = blockIdx.x;  // one cluster per launch
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
        sh.fail = *(volatile int *)&P.status[1] != 0;  // an earlier wait of this call gave up: nothing to do
        for (int b = 0; b < 2; b++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(cl_smem(&sh.bar[b])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = tid; i < C::ROWB / 4; i += TPB) reinterpret_cast<int *>(sh.none)[i] = 0;
    // the barriers exist before any CTA sends to them
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    __syncthreads();

    typename L::Rows x;
    const int g0 = tid / S * S, q0 = tid % S;  // row k of this thread's group: k / S * TPB + g0 + k % S
#pragma unroll
    for (int k = 0; k < R; k++) {
        const int lr = k / S * TPB + g0 + k % S;
#pragma unroll
        for (int i = 0; i < L::WL; i++) x.r[k][i] = lr < nr ? slab[lr * PITCH + i * S + q0] : T(0);
    }
#pragma unroll
    for (int m = 0; m < L::M; m++) {
        x.pos[m] = m * TPB + tid < nr ? rb + m * TPB + tid : -1;
        x.ls[m] = T(0);
    }
    __syncwarp();  // a row's slot is written from here on

    L::columns(P, sh, cl_dyn, x);
    __syncthreads();
    if (!sh.fail) {
        // the pivots and their reciprocals, then the multipliers to the rows'
        // last positions; a pivot row's are scaled by its 1/pivot like the
        // rest of it, and its columns from its own on are in the matrix already
        if (tid < w) {
            const T d = sh.d[tid], inv = cl_zero(d) ? T(1) : T(1) / d;
            sh.inv[tid] = inv;
            if (rank == 0) {
                P.ipiv[c0 + tid] = sh.piv[tid] + P.goff;
                P.dinv[c0 + tid] = inv;
                if (cl_zero(d)) atomicMin(&P.status[0], c0 + tid + 1);
            }
        }
#pragma unroll
        for (int m = 0; m < L::M; m++)
            if (m * TPB + tid < nr) spos[m * TPB + tid] = x.pos[m];
        __syncthreads();
        for (int q = tid; q < nr * CPR; q += TPB) {
            const int lr = q / CPR, ch = q % CPR;
            const int at = spos[lr], have = min(w, at - c0) - ch * VEC;
            if (have <= 0) continue;
            T *dst = P.a + (size_t)at * P.ld + c0 + ch * VEC;
            T v[VEC];
            cl_ld16(cl_smem(slab + lr * PITCH + ch * VEC), v);
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
}

// ---------------------------------------------------------------------------
// The widest slab one cluster of 16 holds in registers (256 threads of 255), by rows:
//   FP64: 64 columns to 4096 rows, 32 to 8192, 16 to 16384
//   FP32: 64 columns to 8192 rows, 32 to 16384, 16 to 32768
// A wider leaf replaces whole levels of the panel recursion (four launches
// each) by rank-1 steps in registers.  Taller panels go to leaf_kernel.
template <typename T, int W>
struct CLeafPick;
template <>
struct CLeafPick<double, 64> {
    static constexpr int S = 4, R = 4, TPB = 256;
};
template <>
struct CLeafPick<double, 32> {
    static constexpr int S = 4, R = 8, TPB = 256;
};
template <>
struct CLeafPick<double, 16> {
    static constexpr int S = 2, R = 8, TPB = 256;
};
template <>
struct CLeafPick<float, 64> {
    static constexpr int S = 4, R = 8, TPB = 256;
};
template <>
struct CLeafPick<float, 32> {
    static constexpr int S = 4, R = 16, TPB = 256;
};
template <>
struct CLeafPick<float, 16> {
    static constexpr int S = 2, R = 16, TPB = 256;
};
template <typename T, int W>
using CLeafPickCfg = CLeafCfg<T, W, CLeafPick<T, W>::S, CLeafPick<T, W>::R, CLeafPick<T, W>::TPB>;

template <typename T, int W>
static constexpr int cl_rows()
{
    return 16 * CLeafPickCfg<T, W>::ROWS;
}

// shared memory and cluster size limits of one instance; true when a cluster of 16 can be resident
template <typename T, int W>
static bool cl_prepare()
{
    using K = CLeafPick<T, W>;
    using C = CLeafPickCfg<T, W>;
    auto kern = cluster_leaf_kernel<T, W, K::S, K::R, K::TPB>;
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
    using C = CLeafPickCfg<T, W>;
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
    return cudaLaunchKernelEx(&cfg, cluster_leaf_kernel<T, W, K::S, K::R, K::TPB>, P);
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

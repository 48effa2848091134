// Left-looking blocked TRSM in one persistent launch (a dependency chain over the 128-row
// blocks of the triangle), for one system and for batches of systems of different sizes.
//
// The reference's left-looking path (special_trsm_template,
// library/src/blas3/rocblas_trsm_kernels.hpp:1164-1456) walks the diagonal blocks on the
// host: per 128-row block j one GEMM tmp = alpha B_j - A_{j,<j} X_{<j} and one GEMM
// X_j = invA_jj tmp, two launches per block.  With few right-hand sides every launch is
// small, so the solve is bound by launch latency.  Here one launch does the whole solve:
//
//   * work items are (block position j in solve order, system, strip of W right-hand sides),
//     enumerated level by level: all systems' items of position 0, then of position 1, ...
//     A CTA claims item ids from a device-side counter in increasing order and works them off
//     in that order, so every item an item depends on (same system and strip, earlier position)
//     was claimed before it by a CTA that is running; the earliest unfinished claimed item
//     therefore never waits on an unfinished one: no deadlock, whatever the residency;
//   * an item computes T = alpha C_b - sum over the finished blocks i of M_{b,i} X_i on DMMA
//     (mma.sync m16n8k8 f64) from a ring of K chunks in shared memory, then X_b = inv(M_bb) T
//     (the caller's or the fused trtri's invA block, its triangle masked), written over C_b, and
//     advances the strip's count of finished blocks (CTA barrier, then st.release.gpu by one
//     thread; blocks of a strip finish in order, so one count per strip is all that is waited on).
//
// The CTA is warp-specialised, because the FP64 tensor pipe (64 FMAs per clock and SM) is what
// the work is bound by and every instruction that the MMA warps spend on copies is time it
// idles: 8 warps only read fragments and issue MMAs, 3 warps copy M (and, after an item's last
// chunk of M, its inverse block) and one warp waits for the strip's count
// (ld.acquire.gpu) and copies X, each through cp.async whose completion arrives on the ring
// slot's barrier.  The copies of M need no flag, so while the CTA waits for the block before its
// own (the dependency chain, which is what few right-hand sides are bound by) that block's
// 128 x 128 tile of M is in shared memory already and one copy of X, two products and one
// store remain between one flag and the next.  The ring runs on across items: the next item's
// copies start while the MMA warps finish the current one.
//
// Measured (one B200, FP64, against the same chain with copies by the MMA warps and 64-column
// strips): 3001 x 77 with invA 716 -> 158 us, 8192 x 512 2.31 -> 1.40 ms (24.5 TFLOP/s), 8192 x
// 8192 23.1 -> 17.6 ms (31.2 TFLOP/s, 0.84 of the tensor pipe's nominal 37.2 and 0.88 of the 35.5
// that cuBLAS DGEMM reaches).  Few right-hand sides are bound by the chain: 5.8 us per block at 8
// columns, of which the two products take 1.6 us.
//
// Every wait is bounded (ChainParams::wait_cycles, about a second); on timeout the kernel
// records error code 4, all roles run out without waiting, and the CTA stops, so a wrong flag
// cannot hang the GPU.
// FP32 systems are staged as FP32 and computed in FP64 (the DMMA path is the one this kernel
// has); the result is rounded to FP32 once.  Complex systems run as real ones of twice the order
// (ChainReal): ztrsm 2048 x 1000, which recursed over one-CTA leaves, 2.30 -> 0.84 ms, and 8192 x
// 2048 25.4 -> 17.9 ms.
//
// The 16 side/uplo/trans/diag cases use the index map of block_solve.cuh: side L solves
// M Y = alpha C with M = op(A), C = B; side R solves M Y = alpha C with M = op(A)^T, C = B^T;
// M(r, c) = tM ? A(c, r) : A(r, c).  Blocks are solved in increasing order when M is lower
// and in decreasing order when M is upper; the K chunks of an item follow the same order.
// Unit diagonals need nothing here: invA already holds the inverse of the unit triangle.
//
// A product with an inverse is not a substitution where something is not finite: the zeros beside
// the triangle turn an infinity of T into NaNs in rows that do not depend on it, and the real
// inverses read a zero diagonal entry as 1.  Systems that a substituting solver would take
// otherwise (ChainParams::subst) must answer as that solver does, so an item of theirs whose X is
// not finite, or whose block has a zero on its diagonal, is solved again from T by substitution
// (chain_substitute).  X finite means that nothing else was in the product: an entry of T or of
// the triangle that is not finite makes the entry of X in its own row so.
#pragma once
#include "gemm_dmma.cuh"
#include "mbarrier.cuh"
#include "timing.hpp"

namespace rb200
{

constexpr int kChainMmaWarps  = 8;
constexpr int kChainCopyWarps = 3; // copies of M and of the inverse blocks
constexpr int kChainMmaThreads  = 32 * kChainMmaWarps;
constexpr int kChainCopyThreads = 32 * kChainCopyWarps;
constexpr int kChainThreads   = kChainMmaThreads + kChainCopyThreads + 32; // + the X warp
constexpr int kChainNB        = 128;

// One system of a variable-size chain launch (sorted by block count, largest first).
template <typename T>
struct ChainSys
{
    const T* A;
    const T* invA; // blocks of 128 x 128, ld 128
    T*       B;
    int64_t  lda, ldb;
    int      k, ncols, nb, ns;
    int      forward, pad;
};

// Tables of a variable-size chain launch for one (tM, side) combination.
template <typename T>
struct ChainVbHeader
{
    const ChainSys<T>* vsys;  // its systems, sorted by nb descending
    const int*         vP;    // vP[i]: prefix sum of ns over vsys[0..i)
    const int*         vcnt;  // vcnt[j]: systems with nb > j
    const int64_t*     vL;    // vL[j]: first item id of level j; vL[maxnb] = its items
    int*               flags; // one per item id
    int                maxnb;
    int                pad;
};

template <typename T>
struct ChainParams
{
    // uniform batch (VB = false): every system has these sizes
    BatchPtr<T>    A;
    int64_t        lda;
    BatchPtr<T>    invA;
    BatchPtr<T>    B;
    int64_t        ldb;
    int            k;       // triangle order
    int            ncols;   // right-hand sides (n for side L, m for side R)
    int            nb, ns;  // blocks, strips
    int            forward; // 1: blocks in increasing order (M lower)
    int64_t        items;   // nb * systems * ns
    int            systems;
    // variable batch (VB = true): the tables of one (tM, side) combination, built on the
    // device by chain_vb_prepass_kernel
    const ChainVbHeader<T>* vhdr;
    Scalar<T>      alpha;   // the caller's alpha
    int            conj = 0; // complex: M's entries are conjugated
    int            unit = 0; // as in BlockSolveParams; only read by a SUBST kernel
    int            subst = 0; // infinities, NaNs and zero diagonals as in a substitution (real types;
                              // complex ones always)
    int            first;   // 1: this solve applies alpha; 0: it applies 1 (a sub-solve after an update)
    // finished blocks per (system, strip), zero at launch: blocks of a strip finish in solve order,
    // so a count serves all their waits; one byte each where flag1 (then at most 255 blocks)
    int*           flags;
    int            flag1 = 0;
    int*           counter; // 8-byte claim counter, zero at launch
    int*           error;   // set to 4 if a wait timed out
    long long      wait_cycles = 1ll << 31; // a flag wait gives up after this many clock cycles
};

__device__ __forceinline__ int chain_ld_acquire(const int* p)
{
    int v;
    asm volatile("ld.global.acquire.gpu.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void chain_st_release(int* p, int v)
{
    asm volatile("st.global.release.gpu.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ int chain_ld_acquire1(const void* p)
{
    int v;
    asm volatile("ld.global.acquire.gpu.u8 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void chain_st_release1(void* p, int v)
{
    asm volatile("st.global.release.gpu.u8 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

template <typename T>
__device__ __forceinline__ void chain_cp_async(uint32_t smem, const T* gmem, bool valid)
{
    const int n = valid ? (int)sizeof(T) : 0;
    if constexpr(sizeof(T) == 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem), "l"(gmem), "r"(n) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem), "l"(gmem), "r"(n) : "memory");
}

// Storage of one real number of T, and whether T is complex.  A complex system is solved as the
// real one of twice the order whose matrix holds [[re, -im], [im, re]] for every entry (rows and
// columns interleaved): C's interleaved storage is then the real right-hand sides as it stands,
// a block of 128 rows is one of 64 complex rows, and the chunks of M keep the complex entries, of
// which a lane reads the component that its row's and column's parity select, with a sign.
template <typename T>
struct ChainReal
{
    using type = T;
    static constexpr int parts = 1;
};
template <typename R>
struct ChainReal<cplx<R>>
{
    using type = R;
    static constexpr int parts = 2;
};

// Shared memory: a ring of stages, each a chunk of M (128 rows o x kBK columns k) and of X (kBK x
// W), then the tile T (128 x W doubles).  Layouts: M [k][o] (KCP = false) or [o][k] (KCP), X
// [k][n] (KCQ = false) or [n][k] (KCQ), elements of type T.  Row pitches keep the fragment reads
// (lanes (g, t) reading element (g, t) or (t, g)) free of bank conflicts: for doubles 4 or 12 mod
// 16 (two half-warp phases), for floats 8 mod 32 where t is the slow index and 4 mod 32 where g is.
// Chunks are 32 deep where four stages fit in shared memory (narrow strips, whose wait for a block
// is covered by the whole tile of M and the start of the inverse in the ring), else 16 deep;
// either depth divides the 128-row blocks, so a chunk never spans two blocks.
template <typename TT, int W, bool KCP, bool KCQ>
struct ChainCfg
{
    using T = typename ChainReal<TT>::type;
    static constexpr int kParts = ChainReal<TT>::parts; // reals per entry of M
    static constexpr int slow_pitch(int n) { return sizeof(T) == 8 ? n + 4 : n + (n % 32 == 0 || n % 32 == 16 ? 8 : 0); }
    static constexpr int pitch_p(int bk) { return KCP ? bk + 4 : slow_pitch(kChainNB); }
    static constexpr int pitch_q(int bk) { return KCQ ? bk + 4 : slow_pitch(W); }
    static constexpr int stage_p(int bk) { return (KCP ? kChainNB : bk) / kParts * pitch_p(bk); }
    static constexpr int stage_q(int bk) { return KCQ ? W * pitch_q(bk) : bk * pitch_q(bk); }
    static constexpr size_t kBytesT = sizeof(double) * (size_t)kChainNB * (W + 4);
    static constexpr size_t kRoom   = 226 * 1024 - kBytesT; // for the ring; the barriers take the rest
    static constexpr int stages(int bk)
    {
        return (int)(kRoom / (sizeof(T) * (size_t)(stage_p(bk) + stage_q(bk))));
    }
    static constexpr int kBK      = stages(32) >= 4 ? 32 : 16;
    static constexpr int kStages  = stages(kBK) < 8 ? stages(kBK) : 8;
    static constexpr int kPitchP  = pitch_p(kBK);
    static constexpr int kPitchQ  = pitch_q(kBK);
    static constexpr int kStageP  = stage_p(kBK);
    static constexpr int kStageQ  = stage_q(kBK);
    static constexpr int kStage   = kStageP + kStageQ; // elements of T
    static constexpr int kPitchT  = W + 4;             // T tile [k = row o][n], doubles
    static constexpr size_t kRing = sizeof(T) * (size_t)kStages * kStage;
    static constexpr size_t kSmem = kRing + kBytesT;
    static_assert(kStages >= 3 && kRing % 16 == 0, "ring");
    // MMA warps: 32 x 32 blocks of the 128 x 64 item, or 16 rows x all W columns of a narrower one
    // (narrower warp rows make the two products of an item equally long for every warp)
    static constexpr int kWarpsN = W == 64 ? 2 : 1;
    static constexpr int kWM     = kChainNB * kWarpsN / kChainMmaWarps; // rows of a warp
    static constexpr int kWN     = W / kWarpsN;                         // columns of a warp
    static constexpr int TM = kWM / 16, TN = kWN / 8;
    // independent accumulators per output tile, so that a warp's MMAs do not wait on one another
    static constexpr int kSplit = TM * TN == 1 ? 4 : TM * TN == 2 ? 2 : 1;
    // The product with the inverse: a row's diagonal term is as a rule the largest of its sum by far,
    // and what an accumulator adds after it is rounded at its magnitude.  So it comes last: the k steps
    // follow the solve's order, or, where a sum is spread over accumulators (kOwn), the term is left out
    // of them and added to their sum at the end in one fused multiply-add.  Error (2-norm) against an
    // 80-bit substitution of order 500, FP64, with ascending steps and with this: forward, 8 columns
    // 0.90 u and 0.71 u (u = 2^-53), 64 columns 0.71 u both; backward 1.88 u and 3.38 u, and 0.71 u.
    static constexpr bool kOwn = kSplit > 1;
};

// One claimed item, resolved for all roles; rows, sizes and leading dimensions in reals.
template <typename T>
struct ChainItem
{
    const T* M;     // M(r0, 0) in A's storage
    const T* inv;   // the block's inverse
    T*       C;     // C(0, c0) in B's storage
    int64_t  lda, ldb;
    int64_t  item;  // < 0: no more items
    int*     flag0; // VB: flag of solve position jj is flag0[vL[jj]]; else the strip's count is
    int64_t  fcell; // flags[fcell]
    int      pos;   // solve position
    int      r0, bs, wv, nb, forward;
    int      klo, khi, ktop; // rows of the finished blocks [klo, khi), chunks counted from ktop when backward
    int      nk, nki;        // chunks of M and of the inverse
};

// C(r0 + o, col) of an item
template <typename T, int PT, bool KCQ>
__device__ __forceinline__ T* chain_caddr(const ChainItem<T>& q, int o, int col)
{
    const int r = q.r0 + o;
    return KCQ       ? q.C + r + (int64_t)col * q.ldb
           : PT == 2 ? q.C + 2 * col + (int64_t)(r >> 1) * q.ldb + (r & 1)
                     : q.C + col + (int64_t)r * q.ldb;
}

// An item's block by substitution from T (Ts, [row][column] with the given pitch), in place and over
// C_b, by the MMA warps.  The reciprocal of the diagonal is multiplied, as the substituting solvers do.
template <typename TT, int W, bool KCP, bool KCQ>
__device__ __noinline__ void chain_substitute(double* Ts, int pitch, const ChainItem<typename ChainReal<TT>::type>& q,
                                              int unit, int conj)
{
    using T = typename ChainReal<TT>::type;
    constexpr int PT = ChainReal<TT>::parts, G = kChainMmaThreads / W;
    const int     rows = q.bs / PT, col = threadIdx.x % W, grp = threadIdx.x / W;
    auto entry = [&](int i, int j, double& re, double& im) {
        const auto* e = KCP ? q.M + i * q.lda + q.r0 + PT * j : q.M + PT * i + (q.r0 / PT + j) * q.lda;
        re = (double)e[0];
        if constexpr(PT == 2)
            im = conj ? -(double)e[1] : (double)e[1];
    };
    // rows solved one after another; a row's value reaches Ts once nobody reads it for an update
    for(int s = 0; s < rows; ++s)
    {
        const int j = q.forward ? s : rows - 1 - s;
        double    dr = 1.0, di = 0.0;
        if(unit != 1)
            entry(j, j, dr, di);
        if(unit == 2 && dr == 0.0 && di == 0.0)
            dr = 1.0;
        double* const row = Ts + PT * j * pitch + col;
        double        xr = row[0], xi = 0.0;
        if constexpr(PT == 2)
        {
            const cplx<double> x = cplx<double>(xr, row[pitch]) * (cplx<double>(1.0) / cplx<double>(dr, di));
            xr = x.x;
            xi = x.y;
        }
        else
            xr *= 1.0 / dr;
        for(int d = 1 + grp; d < rows - s; d += G)
        {
            const int i = q.forward ? j + d : j - d;
            double    mr, mi = 0.0;
            entry(i, j, mr, mi);
            double* const c = Ts + PT * i * pitch + col;
            if constexpr(PT == 2)
            {
                c[0] -= mr * xr - mi * xi;
                c[pitch] -= mr * xi + mi * xr;
            }
            else
                c[0] -= mr * xr;
        }
        asm volatile("barrier.cta.sync 1, %0;" ::"n"(kChainMmaThreads) : "memory");
        if(grp == 0)
        {
            row[0] = xr;
            if constexpr(PT == 2)
                row[pitch] = xi;
        }
    }
    asm volatile("barrier.cta.sync 1, %0;" ::"n"(kChainMmaThreads) : "memory");
    for(int o = grp; o < q.bs && col < q.wv; o += G)
        *chain_caddr<T, PT, KCQ>(q, o, col) = (T)Ts[o * pitch + col];
}

// W right-hand sides per item (8, 16, 32 or 64).  KCP: M's K index is contiguous in memory (tM);
// KCQ: C's row index is contiguous (side L).  VB: the variable-size tables of p describe the items.
// SUBST: ChainParams::subst; a kernel of its own, since the checks and the call cost the others 1 to 4%.
template <typename TT, int W, bool KCP, bool KCQ, bool VB, bool SUBST>
__global__ void __launch_bounds__(kChainThreads, 1) trsm_chain_kernel(ChainParams<TT> p)
{
    using Cfg = ChainCfg<TT, W, KCP, KCQ>;
    using T   = typename Cfg::T;
    constexpr int  PT = Cfg::kParts;
    constexpr bool CX = PT == 2;
    constexpr int TM = Cfg::TM, TN = Cfg::TN, BK = Cfg::kBK, NS = Cfg::kStages, SP = Cfg::kSplit;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T*      ring = reinterpret_cast<T*>(smem_raw);
    double* Ts   = reinterpret_cast<double*>(smem_raw + Cfg::kRing);
    __shared__ ChainItem<T> s_item[2];
    __shared__ uint64_t     full[NS], empty[NS], item_full[2], item_empty[2];
    __shared__ int          s_abort;
    __shared__ int          s_zero[2]; // SUBST: the item's block has a zero on its diagonal

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if(tid == 0)
    {
        s_abort = 0;
        for(int i = 0; i < NS; ++i)
        {
            mbar_init(&full[i], kChainCopyThreads + 32);
            mbar_init(&empty[i], kChainMmaWarps);
        }
        for(int i = 0; i < 2; ++i)
        {
            mbar_init(&item_full[i], 1);
            mbar_init(&item_empty[i], kChainThreads / 32);
        }
    }
    __syncthreads();

    // Bounded waits.  A barrier's owner may itself be waiting for a flag, so barriers wait longer;
    // once a wait ran out (s_abort) every other one returns at once.
    auto aborted = [&]() { return *(volatile int*)&s_abort != 0; };
    auto give_up = [&]() {
        atomicExch(p.error, 4);
        *(volatile int*)&s_abort = 1;
    };
    auto wait_bar = [&](uint64_t* bar, uint32_t parity) {
        if(mbar_try_wait(bar, parity))
            return;
        const long long t0 = clock64();
        while(!mbar_try_wait(bar, parity))
        {
            if(aborted())
                return;
            if(clock64() - t0 > 4 * p.wait_cycles + (1ll << 24))
            {
                give_up();
                return;
            }
        }
    };

    // alpha == 0 anywhere in the call means B := 0 with A unreferenced, also for sub-solves
    // that would otherwise apply 1
    double alpha, alpha_i = 0.0;
    if constexpr(CX)
    {
        const TT ua = p.alpha.get();
        alpha   = (double)ua.x;
        alpha_i = (double)ua.y;
    }
    else
        alpha = (double)p.alpha.get();
    const bool zero = alpha == 0.0 && alpha_i == 0.0;
    if(!zero && !p.first)
    {
        alpha   = 1.0;
        alpha_i = 0.0;
    }

    // claim the next item (one thread)
    auto claim = [&](ChainItem<T>& q) {
        ChainVbHeader<TT> H{};
        if constexpr(VB)
            H = *p.vhdr;
        const int64_t total = VB ? (H.maxnb > 0 ? H.vL[H.maxnb] : 0) : p.items;
        const int64_t item  = aborted() ? total
                                        : (int64_t)atomicAdd(reinterpret_cast<unsigned long long*>(p.counter), 1ull);
        if(item >= total)
        {
            q.item = -1;
            return;
        }
        int      k, ncols, j, strip;
        const T* A;
        T*       B;
        if constexpr(VB)
        {
            static_assert(!CX || !VB, "variable batches are real");
            // level: last j with vL[j] <= item; system: last i < vcnt[j] with vP[i] <= r
            int lo = 0, hi = H.maxnb - 1;
            while(lo < hi)
            {
                const int mid = (lo + hi + 1) >> 1;
                if(H.vL[mid] <= item)
                    lo = mid;
                else
                    hi = mid - 1;
            }
            j = lo;
            const int r = (int)(item - H.vL[j]);
            int       a = 0, z = H.vcnt[j] - 1;
            while(a < z)
            {
                const int mid = (a + z + 1) >> 1;
                if(H.vP[mid] <= r)
                    a = mid;
                else
                    z = mid - 1;
            }
            strip = r - H.vP[a];
            const ChainSys<TT> v = H.vsys[a];
            A = v.A; q.inv = v.invA; B = v.B; q.lda = v.lda; q.ldb = v.ldb;
            k = v.k; ncols = v.ncols; q.nb = v.nb; q.forward = v.forward;
            q.flag0   = H.flags + H.vP[a] + strip;
            q.fcell   = 0;
        }
        else
        {
            strip = (int)(item % p.ns);
            const int64_t js   = item / p.ns;
            const int     sysi = (int)(js % p.systems);
            j = (int)(js / p.systems);
            A     = reinterpret_cast<const T*>(p.A.get(sysi));
            q.inv = reinterpret_cast<const T*>(p.invA.get(sysi));
            B     = reinterpret_cast<T*>(p.B.get(sysi));
            q.lda = p.lda * PT; q.ldb = p.ldb * PT; k = p.k * PT; ncols = p.ncols; q.nb = p.nb;
            q.forward = p.forward;
            q.flag0   = nullptr;
            q.fcell   = (int64_t)sysi * p.ns + strip;
        }
        const int b = q.forward ? j : q.nb - 1 - j;
        q.item = item;
        q.pos  = j;
        q.r0   = b * kChainNB;
        q.bs   = min(kChainNB, k - q.r0);
        q.wv   = min(W, ncols - strip * W);
        q.M    = KCP ? A + (int64_t)(q.r0 / PT) * q.lda : A + q.r0;
        q.inv += (int64_t)b * kChainNB * kChainNB / PT;
        q.C    = KCQ ? B + (int64_t)strip * W * q.ldb : B + strip * W * PT;
        // K rows of the finished blocks: forward [0, r0) ascending; backward [r0 + bs, k)
        // descending, in chunks of BK rows aligned to multiples of BK (never across a block)
        q.klo  = q.forward ? 0 : q.r0 + q.bs;
        q.khi  = q.forward ? q.r0 : k;
        q.ktop = (int)ceil_div(q.khi, BK) * BK;
        q.nk   = zero ? 0 : q.forward ? q.ktop / BK : (q.ktop - q.klo) / BK;
        q.nki  = zero ? 0 : (int)ceil_div(q.bs, BK);
    };
    // barrier of the MMA warps; true in all of them if any saw a wait run out, so that they leave
    // the item loop together, or passed a reason of its own
    auto mma_sync_stop = [&](bool why = false) -> bool {
        int any;
        asm volatile("{\n\t.reg .pred p, q;\n\t"
                     "setp.ne.s32 p, %1, 0;\n\t"
                     "barrier.cta.red.or.pred q, 1, %2, p;\n\t"
                     "selp.s32 %0, 1, 0, q;\n\t}"
                     : "=r"(any)
                     : "r"((int)(why || aborted())), "n"(kChainMmaThreads)
                     : "memory");
        return any != 0;
    };
    auto item_done = [&](int n) {
        __syncwarp();
        if(lane == 0)
            mbar_arrive(&item_empty[n & 1]);
    };

    if(warp >= kChainMmaWarps)
    {
        const bool  copies_m = warp < kChainMmaWarps + kChainCopyWarps;
        uint32_t    st = 0, ph = 1; // ring slot, parity of its last release
        ChainItem<T> q;
        auto slot = [&]() { wait_bar(&empty[st], ph); };
        auto advance = [&]() {
            if(++st == NS)
            {
                st = 0;
                ph ^= 1;
            }
        };
        for(int n = 0;; ++n)
        {
            if(warp == kChainMmaWarps && lane == 0)
            {
                if(n >= 2)
                    wait_bar(&item_empty[n & 1], ((n >> 1) - 1) & 1);
                claim(s_item[n & 1]);
                mbar_arrive(&item_full[n & 1]);
            }
            __syncwarp();
            wait_bar(&item_full[n & 1], (n >> 1) & 1);
            if(aborted())
                break;
            q = s_item[n & 1];
            if(q.item < 0)
                break;
            if(copies_m)
            {
                // ---- chunks of M, then of the inverse --------------------
                // A warp copies every third line of a chunk: a K column (128 rows; four copies
                // per lane) or, K contiguous, 32 / BK rows of BK columns.
                // (complex: half as many lines, of the same number of reals)
                constexpr int kLines = (KCP ? kChainNB * BK / 32 : BK) / PT;
                constexpr int kPer   = KCP ? 1 : kChainNB / 32; // copies per lane and line
                const int     cw  = warp - kChainMmaWarps;
                const int     o0  = KCP ? lane / BK : lane, kk0 = KCP ? lane % BK : 0;
                constexpr int kLineO = KCP ? 32 / BK : 0;
                constexpr uint32_t kDstLine = (uint32_t)sizeof(T) * (KCP ? kLineO : 1) * Cfg::kPitchP;
                const uint32_t dst0 = smem_u32(ring) + (uint32_t)sizeof(T) * (KCP ? o0 * Cfg::kPitchP + kk0 : o0)
                                      + cw * kDstLine;
                const int64_t line = KCP ? kLineO * q.lda : q.lda;
                for(int i = 0; i < q.nk; ++i)
                {
                    const int k0 = q.forward ? i * BK : q.ktop - (i + 1) * BK;
                    slot();
                    uint32_t dst = dst0 + st * (uint32_t)(sizeof(T) * Cfg::kStage);
                    const T* src = (KCP ? q.M + (k0 + kk0) + (int64_t)o0 * q.lda : q.M + o0 + (int64_t)(k0 / PT) * q.lda)
                                   + cw * line;
                    const bool whole = q.bs == kChainNB && k0 + BK <= q.khi;
                    if(whole)
                    {
#pragma unroll 4
                        for(int e = cw; e < kLines; e += kChainCopyWarps)
                        {
#pragma unroll
                            for(int u = 0; u < kPer; ++u)
                                chain_cp_async<T>(dst + u * 32 * (uint32_t)sizeof(T), src + u * 32, true);
                            dst += kChainCopyWarps * kDstLine;
                            src += kChainCopyWarps * line;
                        }
                    }
                    else
                    {
#pragma unroll 1
                        for(int e = cw; e < kLines; e += kChainCopyWarps)
                        {
#pragma unroll
                            for(int u = 0; u < kPer; ++u)
                            {
                                const bool valid = KCP ? (o0 + e * kLineO) * PT < q.bs && k0 + kk0 < q.khi
                                                       : o0 + u * 32 < q.bs && k0 + e * PT < q.khi;
                                chain_cp_async<T>(dst + u * 32 * (uint32_t)sizeof(T), valid ? src + u * 32 : q.M, valid);
                            }
                            dst += kChainCopyWarps * kDstLine;
                            src += kChainCopyWarps * line;
                        }
                    }
                    mbar_arrive_cp_async(&full[st]);
                    advance();
                }
                // inv(M_bb)(o, k) = tM ? invA(k, o) : invA(o, k); rows and columns >= bs are zero (the
                // opposite triangle, which a caller's invA may leave undefined, is masked where the
                // fragments are read)
                for(int i = 0; i < q.nki; ++i)
                {
                    const int k0 = (Cfg::kOwn || q.forward ? i : q.nki - 1 - i) * BK;
                    slot();
                    uint32_t dst = dst0 + st * (uint32_t)(sizeof(T) * Cfg::kStage);
                    if(q.bs == kChainNB)
                    {
                        constexpr int kLine = (KCP ? kLineO : 1) * kChainNB;
                        const T* src = (KCP ? q.inv + (k0 + kk0) + o0 * kChainNB : q.inv + o0 + k0 / PT * kChainNB) + cw * kLine;
#pragma unroll 4
                        for(int e = cw; e < kLines; e += kChainCopyWarps)
                        {
#pragma unroll
                            for(int u = 0; u < kPer; ++u)
                                chain_cp_async<T>(dst + u * 32 * (uint32_t)sizeof(T), src + u * 32, true);
                            dst += kChainCopyWarps * kDstLine;
                            src += kChainCopyWarps * kLine;
                        }
                    }
                    else
#pragma unroll 2
                    for(int e = cw; e < kLines; e += kChainCopyWarps)
                    {
#pragma unroll
                        for(int u = 0; u < kPer; ++u)
                        {
                            const bool valid = KCP ? (o0 + e * kLineO) * PT < q.bs && k0 + kk0 < q.bs
                                                   : o0 + u * 32 < q.bs && k0 + e * PT < q.bs;
                            const T*   src   = KCP ? q.inv + (k0 + kk0) + (o0 + e * kLineO) * kChainNB
                                                   : q.inv + (o0 + u * 32) + (k0 / PT + e) * kChainNB;
                            chain_cp_async<T>(dst + u * 32 * (uint32_t)sizeof(T), valid ? src : q.inv, valid);
                        }
                        dst += kChainCopyWarps * kDstLine;
                    }
                    mbar_arrive_cp_async(&full[st]);
                    advance();
                }
            }
            else
            {
                // ---- chunks of X, each block's after its flag; nothing beside the inverse --------
                constexpr int kFast = KCQ ? BK : W; // lanes run along this dimension
                constexpr int kLanes = kFast < 32 ? kFast : 32;
                constexpr int kStep = 32 / kLanes;  // lines (of the other dimension) per warp copy
                constexpr int kRep  = kFast / kLanes;
                constexpr int kLines = W * BK / kFast;
                const int     f0 = lane % kLanes, l0 = lane / kLanes;
                const uint32_t dst0 = smem_u32(ring)
                                      + (uint32_t)sizeof(T) * (Cfg::kStageP + l0 * Cfg::kPitchQ + f0);
                // a complex strip from the right has its two components as two K lines
                const T* const src0 = q.C + f0 * (KCQ ? 1 : PT);
                auto line_of = [&](int l) -> int64_t { return KCQ || !CX ? l * q.ldb : (l >> 1) * q.ldb + (l & 1); };
                constexpr int kFastStep = KCQ ? 32 : 32 * PT;
                constexpr uint32_t kDstLine = (uint32_t)sizeof(T) * kStep * Cfg::kPitchQ;
                // solve positions [0, done) of the q.pos earlier ones are known finished; one round of
                // loads learns of all that are (VB: of the next 32), so finished blocks cost no round
                // trip each
                int done = 0;
                // (SUBST) the block's diagonal; a complex zero needs no look, it makes the inverse NaN
                constexpr bool kDiag = SUBST && !CX;
                T              diag[kChainNB / 32];
                if constexpr(kDiag)
                {
#pragma unroll
                    for(int u = 0; u < kChainNB / 32; ++u)
                    {
                        const int o = lane + 32 * u;
                        diag[u]     = T(1);
                        if(!zero && !p.unit && o < q.bs)
                            diag[u] = KCP ? q.M[o * q.lda + q.r0 + o] : q.M[o + (q.r0 + o) * q.lda];
                    }
                }
                for(int i = 0; i < q.nk; ++i)
                {
                    const int k0  = q.forward ? i * BK : q.ktop - (i + 1) * BK;
                    const int pos = q.forward ? k0 / kChainNB : q.nb - 1 - k0 / kChainNB;
                    slot();
                    if(pos >= done)
                    {
                        const long long t0 = clock64();
                        for(;;)
                        {
                            if constexpr(VB)
                            {
                                const int      jj    = done + lane;
                                const int      f     = jj < q.pos ? chain_ld_acquire(q.flag0 + p.vhdr->vL[jj]) : 0;
                                const unsigned ready = __ballot_sync(0xffffffffu, f != 0);
                                done += ready == 0xffffffffu ? 32 : __ffs(~ready) - 1;
                            }
                            else
                            {
                                done = p.flag1 ? chain_ld_acquire1(reinterpret_cast<const char*>(p.flags) + q.fcell)
                                               : chain_ld_acquire(p.flags + q.fcell);
                                done = __reduce_min_sync(0xffffffffu, done); // (lanes load the same count)
                            }
                            if(pos < done || __any_sync(0xffffffffu, aborted()))
                                break;
                            if(__any_sync(0xffffffffu, clock64() - t0 > p.wait_cycles))
                            {
                                if(lane == 0)
                                    give_up();
                                break;
                            }
                        }
                        __syncwarp(); // the lanes' acquires order the warp's copies of X below
                    }
                    uint32_t dst = dst0 + st * (uint32_t)(sizeof(T) * Cfg::kStage);
                    const T* base = src0 + (KCQ ? k0 : line_of(k0));
                    if(q.wv == W && k0 + BK <= q.khi)
                    {
#pragma unroll 8
                        for(int e = 0; e < kLines; e += kStep, dst += kDstLine)
                        {
                            const T* src = base + line_of(l0 + e);
#pragma unroll
                            for(int u = 0; u < kRep; ++u)
                                chain_cp_async<T>(dst + u * 32 * (uint32_t)sizeof(T), src + u * kFastStep, true);
                        }
                    }
                    else
                    {
#pragma unroll 1
                        for(int e = 0; e < kLines; e += kStep, dst += kDstLine)
#pragma unroll
                            for(int u = 0; u < kRep; ++u)
                            {
                                const int  f = f0 + u * 32, l = l0 + e;
                                const bool valid = (KCQ ? l : f) < q.wv && k0 + (KCQ ? f : l) < q.khi;
                                chain_cp_async<T>(dst + u * 32 * (uint32_t)sizeof(T),
                                                  valid ? base + line_of(l) + u * kFastStep : q.C, valid);
                            }
                    }
                    mbar_arrive_cp_async(&full[st]);
                    advance();
                }
                for(int i = 0; i < q.nki; ++i)
                {
                    slot();
                    if(kDiag && i + 1 == q.nki)
                    {
                        bool z = false;
#pragma unroll
                        for(int u = 0; u < kChainNB / 32; ++u)
                            z = z || diag[u] == T(0);
                        z = __any_sync(0xffffffffu, z);
                        if(lane == 0)
                            s_zero[n & 1] = z; // read after the last chunk's barrier
                        __syncwarp();
                    }
                    mbar_arrive(&full[st]); // its share of the slot's arrivals
                    advance();
                }
            }
            item_done(n);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        return;
    }

    // ---- the MMA warps -----------------------------------------------------------------------
    // Warps 4..7 take the block rows in opposite order, so that the two warps of a scheduler
    // share the triangle of the inverse evenly.
    const int g = lane >> 2, t = lane & 3;
    const int wn  = Cfg::kWarpsN == 2 ? warp >> 2 : 0;
    const int wm  = warp < 4 ? warp : Cfg::kWarpsN == 2 ? 7 - warp : 11 - warp;
    const int row0 = wm * Cfg::kWM, col0 = wn * Cfg::kWN;
    uint32_t  st = 0, ph = 0;
    auto advance = [&]() {
        __syncwarp();
        if(lane == 0)
            mbar_arrive(&empty[st]);
        if(++st == NS)
        {
            st = 0;
            ph ^= 1;
        }
    };
    // complex: rows o have the parity of g and columns kk that of t, which fixes the component and
    // its sign for the lane
    const int  part = (g ^ t) & 1;
    const bool flip = CX && part && ((g & 1) == 0) != (p.conj != 0);
    auto ldP = [&](const T* sP, int o, int kk) -> double {
        if constexpr(CX)
        {
            const double v = (double)(KCP ? sP[(o >> 1) * Cfg::kPitchP + (kk & ~1) + part]
                                          : sP[(kk >> 1) * Cfg::kPitchP + (o & ~1) + part]);
            return __hiloint2double(__double2hiint(v) ^ (flip ? 0x80000000 : 0), __double2loint(v));
        }
        return (double)(KCP ? sP[o * Cfg::kPitchP + kk] : sP[kk * Cfg::kPitchP + o]);
    };
    auto ldQ = [&](const T* sQ, int n, int kk) -> double {
        return (double)(KCQ ? sQ[n * Cfg::kPitchQ + kk] : sQ[kk * Cfg::kPitchQ + n]);
    };
    auto load_a = [&](double (&fa)[TM][4], const T* sP, int kk, int ku = 4) {
#pragma unroll
        for(int i = 0; i < TM; ++i)
        {
            const int o = row0 + i * 16 + g;
            fa[i][0] = ldP(sP, o, kk);
            fa[i][1] = ldP(sP, o + 8, kk);
            fa[i][2] = ldP(sP, o, kk + ku);
            fa[i][3] = ldP(sP, o + 8, kk + ku);
        }
    };

    for(int n = 0;; ++n)
    {
        wait_bar(&item_full[n & 1], (n >> 1) & 1);
        if(mma_sync_stop())
            break;
        const ChainItem<T> q = s_item[n & 1];
        if(q.item < 0)
            break;
        // C(r0 + o, col) of this thread's output (i, jn, e)
        auto caddr = [&](int o, int col) -> T* { return chain_caddr<T, PT, KCQ>(q, o, col); };
        auto out_o = [&](int i, int e) { return row0 + i * 16 + g + (e >> 1) * 8; };
        auto out_n = [&](int jn, int e) { return col0 + jn * 8 + 2 * t + (e & 1); };

        // ---- 1. acc = M[rows of b, finished rows] X[finished rows, strip] -------------------
        // The sum starts at zero and meets C_b once (C_b in the accumulator would round every
        // small term at C_b's magnitude).  Narrow strips read C_b before the chunks arrive (no
        // other item writes it); wide ones, whose registers are full, after the products.
        constexpr bool kEarlyC = W <= 16;
        auto read_c = [&](double (&c)[TN][4], int i) {
#pragma unroll
            for(int jn = 0; jn < TN; ++jn)
#pragma unroll
                for(int e = 0; e < 4; ++e)
                {
                    const int o = out_o(i, e), col = out_n(jn, e);
                    c[jn][e] = 0.0;
                    if(!zero && o < q.bs && col < q.wv)
                    {
                        const T* src = caddr(o, col);
                        c[jn][e]     = alpha * (double)__ldcg(src);
                        if constexpr(CX) // the other component, times i alpha_i
                            c[jn][e] += (o & 1 ? alpha_i : -alpha_i) * (double)__ldcg(o & 1 ? src - 1 : src + 1);
                    }
                }
        };
        double acc[SP][TM][TN][4], cv[TM][TN][4]; // cv: alpha C_b, then T
        if constexpr(kEarlyC)
#pragma unroll
            for(int i = 0; i < TM; ++i)
                read_c(cv[i], i);
#pragma unroll
        for(int s = 0; s < SP; ++s)
#pragma unroll
            for(int i = 0; i < TM; ++i)
#pragma unroll
                for(int jn = 0; jn < TN; ++jn)
#pragma unroll
                    for(int e = 0; e < 4; ++e)
                        acc[s][i][jn][e] = 0.0;
        auto joined = [&](int i, int jn, int e) { // an output's sum over the accumulators
            if constexpr(SP == 4)
                return (acc[0][i][jn][e] + acc[1][i][jn][e]) + (acc[2][i][jn][e] + acc[3][i][jn][e]);
            else if constexpr(SP == 2)
                return acc[0][i][jn][e] + acc[1][i][jn][e];
            else
                return acc[0][i][jn][e];
        };
        // Fragments are read one k step ahead of the MMAs that use them, for wide strips also
        // across chunks (a narrow one must not hold back a step of the chunk that is there for
        // the next, whose block of X may be microseconds away).
        {
            double fa[2][TM][4], fb[2][TN][2];
            auto   read = [&](int f, int ks) {
                const T*  sP = ring + st * Cfg::kStage;
                const T*  sQ = sP + Cfg::kStageP;
                const int kk = ks * 8 + t;
                load_a(fa[f], sP, kk);
#pragma unroll
                for(int jn = 0; jn < TN; ++jn)
                {
                    const int nn = col0 + jn * 8 + g;
                    fb[f][jn][0] = ldQ(sQ, nn, kk);
                    fb[f][jn][1] = ldQ(sQ, nn, kk + 4);
                }
            };
            auto wait_full = [&]() { wait_bar(&full[st], ph); };
            constexpr bool kAcross = W >= 32;
            constexpr int  KS      = BK / 8;
            static_assert(KS % 2 == 0, "the fragment buffers alternate");
            if(kAcross && q.nk > 0)
            {
                wait_full();
                read(0, 0);
            }
#pragma unroll 1
            for(int c = 0; c < q.nk; ++c)
            {
                if(!kAcross)
                {
                    wait_full();
                    read(0, 0);
                }
#pragma unroll
                for(int ks = 0; ks < KS; ++ks)
                {
                    if(ks + 1 < KS)
                        read((ks + 1) & 1, ks + 1);
                    else
                    {
                        advance();
                        if(kAcross && c + 1 < q.nk)
                        {
                            wait_full();
                            read(0, 0);
                        }
                    }
#pragma unroll
                    for(int i = 0; i < TM; ++i)
#pragma unroll
                        for(int jn = 0; jn < TN; ++jn)
                            dmma_16x8x8(acc[ks % SP][i][jn], fa[ks & 1][i], fb[ks & 1][jn]);
                }
            }
        }

        // ---- 2. T = alpha C_b - sum into shared memory ([row o][col n]), zero outside C_b ---
        // (rows past the block must not reach the product below, whatever X holds)
#pragma unroll
        for(int i = 0; i < TM; ++i)
        {
            if constexpr(!kEarlyC)
                read_c(cv[i], i);
#pragma unroll
            for(int jn = 0; jn < TN; ++jn)
#pragma unroll
                for(int e = 0; e < 4; ++e)
                {
                    const int    o = out_o(i, e), col = out_n(jn, e);
                    const double v = joined(i, jn, e);
#pragma unroll
                    for(int s = 0; s < SP; ++s)
                        acc[s][i][jn][e] = 0.0;
                    cv[i][jn][e] = o < q.bs && col < q.wv ? cv[i][jn][e] - v : 0.0;
                    Ts[o * Cfg::kPitchT + col] = cv[i][jn][e];
                }
            asm volatile("" ::: "memory"); // the next rows' reads stay behind (registers)
        }
        asm volatile("barrier.cta.sync 1, %0;" ::"n"(kChainMmaThreads) : "memory");

        // ---- 3. X_b = inv(M_bb) T: chunks of the inverse through the ring, T resident ---------
        // k steps wholly outside the triangle of this warp's rows are skipped
        // (kOwn) this lane's rows' diagonal entries of the inverse; rows past its last chunk keep 0, as T
        // is there
        double own[2][PT] = {};
        auto   times_inverse = [&](auto ascending) {
            constexpr bool UP = decltype(ascending)::value; // descending: chunks, steps and a step's columns
            // the columns of a step that this lane holds (complex: an entry's two stay together)
            const int     kt = UP ? t : CX ? 6 - (t & ~1) + (t & 1) : 7 - t;
            constexpr int ku = UP ? 4 : -4;
#pragma unroll 1
            for(int c = 0; c < q.nki; ++c)
            {
                const T*  sP = ring + st * Cfg::kStage;
                const int k0 = (UP ? c : q.nki - 1 - c) * BK; // row of T
                wait_bar(&full[st], ph);
                if constexpr(Cfg::kOwn)
                {
                    static_assert(TM == 1 && BK % Cfg::kWM == 0, "a warp's rows are in one chunk");
                    if(k0 == row0 / BK * BK)
#pragma unroll
                        for(int r = 0; r < 2; ++r)
                        {
                            const int o = row0 + g + 8 * r, kk = (o - k0) / PT * PT; // the entry's first column
#pragma unroll
                            for(int x = 0; x < PT; ++x)
                                own[r][x] = (double)(KCP ? sP[o / PT * Cfg::kPitchP + kk + x]
                                                         : sP[kk / PT * Cfg::kPitchP + o / PT * PT + x]);
                        }
                }
#pragma unroll
                for(int u = 0; u < BK / 8; ++u)
                {
                    const int ks = UP ? u : BK / 8 - 1 - u, kb = k0 + ks * 8;
                    if(q.forward ? kb > row0 + Cfg::kWM - 1 : kb + 7 < row0)
                        continue;
                    double fa[TM][4], fb[TN][2];
                    load_a(fa, sP, ks * 8 + kt, ku);
                    // entries outside the triangle, in the k steps that touch the warp's rows
                    if(q.forward ? kb + 7 > row0 - Cfg::kOwn : kb < row0 + Cfg::kWM - 1 + Cfg::kOwn)
#pragma unroll
                        for(int i = 0; i < TM; ++i)
#pragma unroll
                            for(int e = 0; e < 4; ++e)
                            {
                                const int o = out_o(i, 2 * (e & 1)) / PT, kr = (kb + kt + ku * (e >> 1)) / PT;
                                if(q.forward ? kr > o - Cfg::kOwn : kr < o + Cfg::kOwn)
                                    fa[i][e] = 0.0;
                            }
#pragma unroll
                    for(int jn = 0; jn < TN; ++jn)
                    {
                        const int nn = col0 + jn * 8 + g;
                        fb[jn][0] = Ts[(kb + kt) * Cfg::kPitchT + nn];
                        fb[jn][1] = Ts[(kb + kt + ku) * Cfg::kPitchT + nn];
                    }
#pragma unroll
                    for(int i = 0; i < TM; ++i)
#pragma unroll
                        for(int jn = 0; jn < TN; ++jn)
                            dmma_16x8x8(acc[u % SP][i][jn], fa[i], fb[jn]);
                }
                advance();
            }
        };
        if(Cfg::kOwn || q.forward)
            times_inverse(std::true_type{});
        else
            times_inverse(std::false_type{});

        // ---- 4. X_b over C_b, then release the item's flag ---------------------------------
        const bool live = !aborted();
        bool       redo = false; // (SUBST) not what a substitution gives
        if constexpr(SUBST && !CX)
            redo = q.nki > 0 && s_zero[n & 1];
#pragma unroll
        for(int i = 0; i < TM; ++i)
#pragma unroll
            for(int jn = 0; jn < TN; ++jn)
#pragma unroll
                for(int e = 0; e < 4; ++e)
                {
                    const int o = out_o(i, e), col = out_n(jn, e);
                    double    v = joined(i, jn, e);
                    if constexpr(Cfg::kOwn)
                        if(q.nki > 0)
                        {
                            const double T_o = cv[i][jn][e];
                            if constexpr(CX)
                            {
                                // [[re, -im], [im, re]] times the row's pair of T
                                const double im = (o & 1) == 0 ? -own[e >> 1][1] : own[e >> 1][1];
                                v = fma(p.conj ? -im : im, Ts[(o ^ 1) * Cfg::kPitchT + col], v);
                            }
                            else if(!is_finite(T_o))
                                v = 0.0; // the 0 in the term's place made it NaN
                            v = fma(own[e >> 1][0], T_o, v);
                        }
                    if constexpr(SUBST)
                        redo = redo || !is_finite(v); // (0 outside C_b unless something in it is not)
                    if(live && o < q.bs && col < q.wv)
                        *caddr(o, col) = (T)v;
                }
        // all of X_b is written (and T free for the next item) once every MMA warp is here
        if constexpr(!SUBST)
        {
            if(mma_sync_stop())
                break;
        }
        else if(mma_sync_stop(redo))
        {
            if(mma_sync_stop())
                break;
            chain_substitute<TT, W, KCP, KCQ>(Ts, Cfg::kPitchT, s_item[n & 1], p.unit, p.conj);
            if(mma_sync_stop())
                break;
        }
        if(tid == 0)
        {
            if constexpr(VB)
                chain_st_release(p.vhdr->flags + q.item, 1);
            else if(p.flag1)
                chain_st_release1(reinterpret_cast<char*>(p.flags) + q.fcell, q.pos + 1);
            else
                chain_st_release(p.flags + q.fcell, q.pos + 1);
        }
        item_done(n);
    }
}

// Blocks, strips and the workspace of one uniform chain solve: the strips' counts, then (8-byte
// aligned) the 8-byte claim counter and a spare error word.  The counts take one word per 128-row
// block and 64-column strip, whatever the width: as words where that is enough for the strips, else
// (narrow strips of a few blocks) as bytes.
struct ChainShape
{
    int     nb, ns, w;
    int64_t items;
    int64_t words;  // of the counts' space
    int     flag1;  // counts are bytes
};

inline ChainShape chain_shape(int k, int ncols, int batch, int w)
{
    ChainShape c;
    c.w     = w;
    c.nb    = (int)ceil_div(k, kChainNB);
    c.ns    = (int)ceil_div(ncols, w);
    c.items = (int64_t)batch * c.nb * c.ns;
    c.words = (int64_t)batch * c.nb * ceil_div(ncols, 64);
    c.flag1 = (int64_t)batch * c.ns > c.words; // then nb < 8, and the counts fit as bytes
    if(c.flag1 && (int64_t)batch * c.ns > 4 * c.words)
        return chain_shape(k, ncols, batch, 64); // (one block of 8-column strips)
    return c;
}

inline size_t chain_workspace_bytes(const ChainShape& c)
{
    return ((size_t)c.words * sizeof(int) + 7) / 8 * 8 + 16;
}

// cluster2: the grid as clusters of two CTAs (placement only; the kernel uses no cluster
// feature), for an even grid
template <typename T, int W, bool KCP, bool KCQ, bool VB>
static void launch_chain_cfg(const ChainParams<T>& p, int sms, int64_t max_items, cudaStream_t s,
                             bool cluster2 = false)
{
    using Cfg = ChainCfg<T, W, KCP, KCQ>;
    auto kern = trsm_chain_kernel<T, W, KCP, KCQ, VB, is_cplx<T>::value>;
    if constexpr(!is_cplx<T>::value && !VB)
        if(p.subst)
            kern = trsm_chain_kernel<T, W, KCP, KCQ, VB, true>;
    cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::kSmem);
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kChainThreads, Cfg::kSmem);
    const int64_t grid = std::max<int64_t>(1, std::min<int64_t>(max_items, (int64_t)sms * std::max(per_sm, 1)));
    // algorithmic work (uniform batch): k * k * ncols per system, the trsm flop count
    const double work = VB ? 0.0 : (is_cplx<T>::value ? 4.0 : 1.0) * p.systems * p.k * (double)p.k * p.ncols;
    TimedLaunch tl(KernelClass::chain, s, work);
    if(cluster2 && grid % 2 == 0)
    {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim          = dim3((unsigned)grid);
        cfg.blockDim         = dim3(kChainThreads);
        cfg.dynamicSmemBytes = Cfg::kSmem;
        cfg.stream           = s;
        cudaLaunchAttribute at[1];
        at[0].id               = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = 2;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs    = at;
        cfg.numAttrs = 1;
        cudaLaunchKernelEx(&cfg, kern, p);
    }
    else
        kern<<<(unsigned)grid, kChainThreads, Cfg::kSmem, s>>>(p);
}

template <typename T, int W, bool VB>
void launch_chain_w(const ChainParams<T>& p, bool kcp, bool kcq, int sms, int64_t max_items,
                           cudaStream_t s, bool cluster2 = false)
{
    if(kcp && kcq)
        launch_chain_cfg<T, W, true, true, VB>(p, sms, max_items, s, cluster2);
    else if(kcp)
        launch_chain_cfg<T, W, true, false, VB>(p, sms, max_items, s, cluster2);
    else if(kcq)
        launch_chain_cfg<T, W, false, true, VB>(p, sms, max_items, s, cluster2);
    else
        launch_chain_cfg<T, W, false, false, VB>(p, sms, max_items, s, cluster2);
}

// instantiated in chain_kernels.cu
extern template void launch_chain_w<double, 8, false>(const ChainParams<double>&, bool, bool, int, int64_t, cudaStream_t, bool);
extern template void launch_chain_w<double, 16, false>(const ChainParams<double>&, bool, bool, int, int64_t, cudaStream_t, bool);
extern template void launch_chain_w<double, 32, false>(const ChainParams<double>&, bool, bool, int, int64_t, cudaStream_t, bool);
extern template void launch_chain_w<double, 64, false>(const ChainParams<double>&, bool, bool, int, int64_t, cudaStream_t, bool);
extern template void launch_chain_w<double, 32, true>(const ChainParams<double>&, bool, bool, int, int64_t, cudaStream_t, bool);
extern template void launch_chain_w<double, 64, true>(const ChainParams<double>&, bool, bool, int, int64_t, cudaStream_t, bool);
extern template void launch_chain_w<float, 8, false>(const ChainParams<float>&, bool, bool, int, int64_t, cudaStream_t, bool);
extern template void launch_chain_w<float, 16, false>(const ChainParams<float>&, bool, bool, int, int64_t, cudaStream_t, bool);
extern template void launch_chain_w<float, 32, false>(const ChainParams<float>&, bool, bool, int, int64_t, cudaStream_t, bool);
extern template void launch_chain_w<float, 64, false>(const ChainParams<float>&, bool, bool, int, int64_t, cudaStream_t, bool);
extern template void launch_chain_w<float, 32, true>(const ChainParams<float>&, bool, bool, int, int64_t, cudaStream_t, bool);
extern template void launch_chain_w<float, 64, true>(const ChainParams<float>&, bool, bool, int, int64_t, cudaStream_t, bool);

extern template void launch_chain_w<cplx<double>, 8, false>(const ChainParams<cplx<double>>&, bool, bool, int, int64_t, cudaStream_t, bool);
extern template void launch_chain_w<cplx<double>, 16, false>(const ChainParams<cplx<double>>&, bool, bool, int, int64_t, cudaStream_t, bool);
extern template void launch_chain_w<cplx<double>, 32, false>(const ChainParams<cplx<double>>&, bool, bool, int, int64_t, cudaStream_t, bool);
extern template void launch_chain_w<cplx<double>, 64, false>(const ChainParams<cplx<double>>&, bool, bool, int, int64_t, cudaStream_t, bool);
extern template void launch_chain_w<cplx<float>, 8, false>(const ChainParams<cplx<float>>&, bool, bool, int, int64_t, cudaStream_t, bool);
extern template void launch_chain_w<cplx<float>, 16, false>(const ChainParams<cplx<float>>&, bool, bool, int, int64_t, cudaStream_t, bool);
extern template void launch_chain_w<cplx<float>, 32, false>(const ChainParams<cplx<float>>&, bool, bool, int, int64_t, cudaStream_t, bool);
extern template void launch_chain_w<cplx<float>, 64, false>(const ChainParams<cplx<float>>&, bool, bool, int, int64_t, cudaStream_t, bool);
} // namespace rb200

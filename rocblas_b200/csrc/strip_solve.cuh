// One-CTA triangular solve of a strip of right-hand sides, real types, for small and batched
// systems (complex types: block_solve.cuh, whose index map of the 16 side/uplo/trans/diag
// combinations this file shares).
//
// Replaces the reference's small and substitution kernels
// (library/src/blas3/rocblas_trsm_kernels.hpp: rocblas_trsm_small_right_device :1962-2227,
// rocblas_trsm_small_left_device :2359-2560, ..._sharedB :2562-2780, the blocked
// forward/backward substitution :3059-3261 and its host loop :3263-3515):
//   side L:  op(A) X = alpha B          ->  M Y = alpha C with M = op(A),   C = B,   Y = X
//   side R:  X op(A) = alpha B          ->  M Y = alpha C with M = op(A)^T, C = B^T, Y = X^T
// and an upper M becomes lower by reversing the rows (i -> k-1-i).
//
// The solve is done transposed on the FP64 tensor path, Y^T M^T = alpha C^T, with the right-hand
// sides in the registers of the warp that owns them: an mma.sync m8n8k4 accumulator holds, for 8
// right-hand sides (lane / 4) and 8 rows of C, the rows 2t and 2t+1 (t = lane % 4) in each lane,
// and since the order of a product's inner index is free, those two registers are as they stand
// the left operands of the two m8n8k4 products over the same 8 rows.  So a solved tile feeds the
// updates of all rows below without a shuffle or a trip through shared memory, no warp waits for
// another one's columns, and what was a substitution by one warp of eight is a chain of MMAs in
// each:
//   * the rows are cut into super-blocks of 8 RT rows (acc[RT][2] in registers);
//   * M is staged in panels of 8 RT rows x 32 columns through a cp.async ring shared by the CTA's
//     four warps, as 8 x 8 tiles whose rows are swizzled so that copies along either direction and
//     the fragment reads (one 16- or 8-byte read per lane and tile) do not collide;
//   * panels left of the super-block's diagonal update it with the finished rows, whose values
//     each lane reads back from where it wrote them in C;
//   * a diagonal panel's four 8 x 8 tiles are inverted by each warp (lane = column, 28 FMAs) and
//     every tile of the solve is then X = T inv^T, one more product, followed by the updates of
//     the super-block's rows below.  Where that X is not finite (as it is where the inverse or the
//     right-hand side is not, or where terms of the product overflow that a substitution would cancel
//     before it divides) the tile is substituted row by row instead, so that an infinity or NaN
//     reaches exactly the rows that it reaches in a substitution.
// FP32 systems are staged as FP32 and computed in FP64.
//
// Measured (one B200, against the solver with the strip in shared memory and one-warp
// substitutions; passes with the copy of the right-hand sides): 4096 systems of 128 x 32 in FP64
// 515 -> 209 us, 20,000 uneven systems 4.39 -> 2.00 ms, one 96 x 24 system 18.5 -> 12.3-14.3 us.  What
// bounds the uniform batch is the L1 data pipe (75% busy; DRAM 40%, DMMA 40%): every warp reads the
// whole triangle for its 8 right-hand sides.
#pragma once
#include <type_traits>

#include "common.cuh"
#include "mbarrier.cuh"
#include "mma_f64.cuh"

namespace rb200
{

// One system (or a uniform batch of systems).
template <typename T>
struct BlockSolveParams
{
    int         m, n, k;        // B is m x n; A is k x k
    int         side_left;
    int         tM;             // M(i,j) = tM ? A(j,i) : A(i,j)
    int         rev;            // M upper: rows reversed
    int         unit;           // complex, 2: a zero diagonal entry is read as 1
    int         conj;           // M's entries are conjugated (complex trans C)
    BatchPtr<T> A;
    int64_t     lda;
    BatchPtr<T> B;
    int64_t     ldb;
    Scalar<T>   ualpha;         // the caller's alpha
    int         first;          // 1: this solve applies ualpha; 0: it applies 1
    int         batch_base;
};

constexpr int kSsW       = 32;  // right-hand sides per CTA
constexpr int kSsThreads = 128; // 8 right-hand sides per warp
constexpr int kSsPanel   = 32;  // columns of M per panel
constexpr int kSsMaxK    = 512;
// Super-blocks of 64 rows, two panels in the ring, registers for four CTAs per SM, measured side by
// side: 211 us for 4096 systems of 128 x 32 and 2010 us for 20,000 uneven ones (five CTAs 224 and
// 2139; 128 rows, which leave three, 242 and 2350; three and four panels were no faster).
constexpr int kSsRT   = 8;
constexpr int kSsNS   = 2;
constexpr int kSsCtas = 4;

template <typename T, int RT, int NS>
struct SsCfg
{
    static constexpr int kRows  = 8 * RT;
    static constexpr int kStage = RT * 4 * 64; // elements of one panel
    static constexpr size_t kSmem
        = sizeof(double) * (size_t)(kSsThreads / 32 * 4 * 64) + sizeof(T) * (size_t)NS * kStage;
};

// Element (i, j) of an 8 x 8 tile: rows of four pairs, the pairs of a row permuted by the row.
template <typename T>
__device__ __forceinline__ constexpr int ss_swizzle(int i)
{
    return sizeof(T) == 8 ? i >> 1 : i >> 2;
}
template <typename T>
__device__ __forceinline__ constexpr int ss_elem(int i, int j)
{
    return i * 8 + (((j >> 1) ^ ss_swizzle<T>(i)) << 1) + (j & 1);
}

// lane (g, t)'s pair (row g, columns 2t and 2t + 1) of a tile
__device__ __forceinline__ void ss_pair(const double* tile, int pair, double& b0, double& b1)
{
    const double2 v = *reinterpret_cast<const double2*>(tile + pair);
    b0 = v.x;
    b1 = v.y;
}
__device__ __forceinline__ void ss_pair(const float* tile, int pair, double& b0, double& b1)
{
    const float2 v = *reinterpret_cast<const float2*>(tile + pair);
    b0 = (double)v.x;
    b1 = (double)v.y;
}

// One strip: columns s0 .. s0 + 31 (of ncols) of C.  NS: panels in the ring.
template <typename T, int RT, int NS>
__device__ __forceinline__ void strip_solve(const T* A, int64_t lda, T* B, int64_t ldb, int k, int side_left, int tM,
                                            int rev, int unit, double alpha, int s0, int ncols,
                                            unsigned char* smem_raw)
{
    using Cfg = SsCfg<T, RT, NS>;
    constexpr int R = Cfg::kRows, NP = R / kSsPanel; // panels across a super-block
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    double* const inv  = reinterpret_cast<double*>(smem_raw) + warp * 4 * 64; // this warp's inverses
    T* const      ring = reinterpret_cast<T*>(smem_raw + sizeof(double) * (size_t)(kSsThreads / 32 * 4 * 64));

    const int  W    = min(kSsW, ncols - s0);
    const int  col  = warp * 8 + g;
    const bool live = warp * 8 < W; // the warp has right-hand sides
    const bool ok   = col < W;

    // C'(i, col), rows reversed when rev: C0[i * dr]
    const int64_t bdr = side_left ? 1 : ldb, bdc = side_left ? ldb : 1;
    T* const      C0 = B + (s0 + col) * bdc + (rev ? (int64_t)(k - 1) * bdr : 0);
    const int64_t dr = rev ? -bdr : bdr;
    if(alpha == 0.0)
    {
        // C := 0 without reading A or C (rocblas_trsm_imp.hpp:154-157 semantics)
        if(ok)
            for(int i = t; i < k; i += 4)
                C0[i * dr] = T(0);
        return;
    }
    // M'(i, j), the reversed lower orientation: M0[i dI + j dJ]
    const int64_t  sgn = rev ? -1 : 1;
    const int64_t  dI = (tM ? lda : 1) * sgn, dJ = (tM ? 1 : lda) * sgn;
    const T* const M0 = A + (rev ? (int64_t)(k - 1) * (1 + lda) : 0);

    const int nsb = (k + R - 1) / R; // super-blocks

    // ---- panel copies: panel (I, J, p) is rows I R .. + R, columns J R + 32 p .. + 32 -------------
    // A diagonal panel (J == I) keeps the rows from its own on, the triangle zero-filled above the
    // diagonal; the diagonal itself is copied unless it is a unit one.
    struct Pos
    {
        int I, J, p;
    };
    auto step = [&](Pos& q) {
        ++q.p;
        if(q.p == NP || (q.J == q.I && q.I * R + q.p * kSsPanel >= k))
        {
            q.p = 0;
            if(++q.J > q.I)
            {
                q.J = 0;
                ++q.I;
            }
        }
    };
    auto cp = [&](uint32_t dst, const T* src, bool valid) {
        const int n = valid ? (int)sizeof(T) : 0;
        const T*  s = valid ? src : A;
        if constexpr(sizeof(T) == 8)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(s), "r"(n) : "memory");
        else
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(s), "r"(n) : "memory");
    };
    auto copy_panel = [&](int stage, const Pos& q) {
        const uint32_t base = smem_u32(ring + stage * Cfg::kStage);
        const bool     diag = q.J == q.I;
        const int      j0 = q.J * R + q.p * kSsPanel, i0 = q.I * R;
        const int      first = diag ? q.p * kSsPanel : 0; // first row of the panel that exists
        const int      last  = min(R, k - i0);            // rows of the super-block
        const int      pad   = (last + 7) & ~7;           // zero-filled to whole tiles
        if(!tM)
        {
            // lanes along the rows: rows tid (+ 128 ..), all 32 columns
            for(int i = first + tid; i < pad; i += kSsThreads)
            {
                const uint32_t d0 = base + (uint32_t)sizeof(T) * ((i >> 3) * 4 * 64 + (i & 7) * 8);
                const int      sw = ss_swizzle<T>(i & 7);
                const int      lim = i >= last ? 0 : min(kSsPanel, (diag ? i - q.p * kSsPanel + (unit ? 0 : 1) : k - j0));
                const T*       src = M0 + (i0 + i) * dI + j0 * dJ;
#pragma unroll 8
                for(int j = 0; j < kSsPanel; ++j, src += dJ)
                    cp(d0 + (uint32_t)sizeof(T) * ((j >> 3) * 64 + ((((j >> 1) & 3) ^ sw) << 1) + (j & 1)), src, j < lim);
            }
        }
        else
        {
            // lanes along the columns: rows warp, warp + 4, ..
#pragma unroll 8
            for(int i = first + warp; i < pad; i += kSsThreads / 32)
            {
                const bool valid = i < last && (diag ? lane < i - q.p * kSsPanel + (unit ? 0 : 1) : j0 + lane < k);
                cp(base + (uint32_t)sizeof(T) * ((i >> 3) * 4 * 64 + (lane >> 3) * 64 + ss_elem<T>(i & 7, lane & 7)),
                   M0 + (i0 + i) * dI + (j0 + lane) * dJ, valid);
            }
        }
    };

    Pos ld{0, 0, 0}; // next panel to copy
    int ls = 0;      // its stage
    auto copy_next = [&]() {
        if(ld.I < nsb)
        {
            copy_panel(ls, ld);
            step(ld);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        ls = ls + 1 == NS ? 0 : ls + 1;
    };
    int cs = 0; // stage of the panel to compute
    // the next panel has landed, and its predecessor's stage is free for the copies
    auto next_panel = [&]() -> const T* {
        asm volatile("cp.async.wait_group %0;" ::"n"(NS - 2) : "memory");
        __syncthreads();
        copy_next();
        const T* s = ring + cs * Cfg::kStage;
        cs = cs + 1 == NS ? 0 : cs + 1;
        return s;
    };
#pragma unroll
    for(int s = 0; s < NS - 1; ++s)
        copy_next();

    const int pairT = g * 8 + ((t ^ ss_swizzle<T>(g)) << 1);      // this lane's pair of a tile of M
    const int pairD = g * 8 + ((t ^ ss_swizzle<double>(g)) << 1); // ... of an inverse
    double    acc[RT][2];
    // acc[r] += x M(r, .)^T over the tiles r of one 8-column step, four at a time; tiles past the
    // super-block's rows hold nothing
    auto update = [&](double x0, double x1, const T* tiles, auto r_first, int nrt) {
        constexpr int R0 = decltype(r_first)::value;
#pragma unroll
        for(int r = R0; r < RT; r += 4)
            if(r < nrt)
            {
                double b[4][2];
#pragma unroll
                for(int u = 0; u < 4; ++u)
                    if(r + u < RT)
                        ss_pair(tiles + (r + u) * 4 * 64 + pairT, 0, b[u][0], b[u][1]);
#pragma unroll
                for(int u = 0; u < 4; ++u)
                    if(r + u < RT)
                        dmma_8x8x4(acc[r + u], x0, b[u][0]);
#pragma unroll
                for(int u = 0; u < 4; ++u)
                    if(r + u < RT)
                        dmma_8x8x4(acc[r + u], x1, b[u][1]);
            }
    };

    for(int I = 0; I < nsb; ++I)
    {
        const int i0 = I * R, rows = min(R, k - i0), nrt = (rows + 7) / 8;
        // sums of M X over the solved rows; a row's sum gives way to its solution
#pragma unroll
        for(int r = 0; r < RT; ++r)
            acc[r][0] = acc[r][1] = 0.0;
        // ---- panels left of the diagonal ------------------------------------------------------------
        for(int j = 0; j < I * NP; ++j)
        {
            double   x[4][2]; // X^T of the panel's rows: what this lane wrote
            const T* c = C0 + (j * kSsPanel + 2 * t) * dr;
#pragma unroll
            for(int q = 0; q < 4; ++q, c += 8 * dr)
            {
                x[q][0] = ok ? (double)c[0] : 0.0;
                x[q][1] = ok ? (double)c[dr] : 0.0;
            }
            const T* S = next_panel();
            if(live)
#pragma unroll
                for(int q = 0; q < 4; ++q)
                    update(x[q][0], x[q][1], S + q * 64, std::integral_constant<int, 0>{}, nrt);
        }
        // ---- diagonal panels -----------------------------------------------------------------------
        auto diagonal = [&](auto p_const) {
            constexpr int P = decltype(p_const)::value;
            if(P * kSsPanel >= rows)
                return;
            // alpha C' of the panel's rows: the sums start at zero and meet it once (in the
            // accumulator it would round every small term at its own magnitude)
            double cv[4][2];
            {
                const T*  c   = C0 + (i0 + P * kSsPanel + 2 * t) * dr;
                const int lim = ok ? k - i0 - P * kSsPanel - 2 * t : 0; // rows left
#pragma unroll
                for(int q = 0; q < 4; ++q, c += 8 * dr)
                {
                    cv[q][0] = 8 * q < lim ? alpha * (double)c[0] : 0.0;
                    cv[q][1] = 8 * q + 1 < lim ? alpha * (double)c[dr] : 0.0;
                }
            }
            const T* S = next_panel();
            if(!live)
                return;
            // inverses of the four diagonal tiles: lane = (tile, column)
            {
                const int q = lane >> 3, c = lane & 7;
                const T*  D = S + ((P * 4 + q) * 4 + q) * 64;
                // a unit diagonal and padding rows: 1
                const double d  = unit || P * kSsPanel + lane >= rows ? 1.0 : (double)D[ss_elem<T>(c, c)];
                const double rd = 1.0 / d;
                double       s[8];
#pragma unroll
                for(int i = 0; i < 8; ++i)
                    s[i] = i == c ? 1.0 : 0.0;
#pragma unroll
                for(int j = 0; j < 8; ++j)
                {
                    s[j] *= __shfl_sync(0xffffffffu, rd, (lane & 24) | j);
#pragma unroll
                    for(int i = j + 1; i < 8; ++i)
                        s[i] -= (double)D[ss_elem<T>(i, j)] * s[j];
                }
                __syncwarp(); // the previous panel's inverses are read
#pragma unroll
                for(int i = 0; i < 8; ++i)
                    inv[q * 64 + ss_elem<double>(i, c)] = s[i];
                __syncwarp();
            }
            auto solve_tile = [&](auto q_const) {
                constexpr int Q = decltype(q_const)::value, s = P * 4 + Q;
                if(s >= nrt)
                    return;
                double       x[2] = {0.0, 0.0};
                const double T0 = cv[Q][0] - acc[s][0], T1 = cv[Q][1] - acc[s][1];
                {
                    double b0, b1;
                    ss_pair(inv + Q * 64 + pairD, 0, b0, b1);
                    dmma_8x8x4(x, T0, b0);
                    dmma_8x8x4(x, T1, b1);
                }
                if(!__all_sync(0xffffffffu, is_finite(x[0]) && is_finite(x[1])))
                {
                    // row by row: the lane that holds row j scales it and hands it to its column's
                    // other lanes
                    const T* D = S + (s * 4 + Q) * 64;
                    x[0] = T0;
                    x[1] = T1;
#pragma unroll 1
                    for(int j = 0; j < 8; ++j)
                    {
                        const double d = unit || s * 8 + j >= rows ? 1.0 : (double)D[ss_elem<T>(j, j)];
                        if(t == j >> 1)
                        {
                            if(j & 1)
                                x[1] *= 1.0 / d;
                            else
                                x[0] *= 1.0 / d;
                        }
                        const double xj = __shfl_sync(0xffffffffu, j & 1 ? x[1] : x[0], (lane & 28) | (j >> 1));
                        if(2 * t > j)
                            x[0] -= (double)D[ss_elem<T>(2 * t, j)] * xj;
                        if(2 * t + 1 > j)
                            x[1] -= (double)D[ss_elem<T>(2 * t + 1, j)] * xj;
                    }
                }
                acc[s][0] = x[0];
                acc[s][1] = x[1];
                if constexpr(s + 1 < RT)
                    update(x[0], x[1], S + Q * 64, std::integral_constant<int, s + 1>{}, nrt);
            };
            solve_tile(std::integral_constant<int, 0>{});
            solve_tile(std::integral_constant<int, 1>{});
            solve_tile(std::integral_constant<int, 2>{});
            solve_tile(std::integral_constant<int, 3>{});
        };
        diagonal(std::integral_constant<int, 0>{});
        if constexpr(NP > 1)
            diagonal(std::integral_constant<int, 1>{});
        if constexpr(NP > 2)
        {
            diagonal(std::integral_constant<int, 2>{});
            diagonal(std::integral_constant<int, 3>{});
        }
        // ---- Y over C -------------------------------------------------------------------------------
        {
            T*        c   = C0 + (i0 + 2 * t) * dr;
            const int lim = ok ? k - i0 - 2 * t : 0;
#pragma unroll
            for(int r = 0; r < RT; ++r, c += 8 * dr)
            {
                if(8 * r < lim)
                    c[0] = (T)acc[r][0];
                if(8 * r + 1 < lim)
                    c[dr] = (T)acc[r][1];
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// CTAS: resident CTAs per SM that the registers are cut for.
template <typename T, int RT, int NS, int CTAS>
__global__ void __launch_bounds__(kSsThreads, CTAS) strip_solve_kernel(BlockSolveParams<T> p)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int batch = p.batch_base + blockIdx.y;
    // alpha == 0 anywhere in the call means B := 0 with A unreferenced, also for the
    // sub-solves of the blocked path that would otherwise apply 1
    const double ua    = (double)p.ualpha.get();
    const double alpha = ua == 0.0 ? 0.0 : (p.first ? ua : 1.0);
    strip_solve<T, RT, NS>(p.A.get(batch), p.lda, p.B.get(batch), p.ldb, p.k, p.side_left, p.tM, p.rev, p.unit, alpha,
                           blockIdx.x * kSsW, p.side_left ? p.n : p.m, smem_raw);
}

} // namespace rb200

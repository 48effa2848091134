// Inversion of the diagonal blocks of a triangular matrix, one CTA per block of up to 128.
//
// Replaces the reference's invA construction for TRSM (rocblas_trtri_trsm_template,
// library/src/blas3/trtri_trsm.hpp:110-381: 16x16 trtri kernels, three rounds of
// strided-batched GEMM merges 32->64->128, a separate fill kernel for the unused
// triangle and a remainder trtri) with a single fused kernel: the block (at most 128 x 128,
// padded with the identity) is staged in shared memory in lower orientation (an upper block U
// is handled as the lower block J U J, J the exchange matrix), its eight 16 x 16 diagonal
// tiles are inverted by one warp each (lane = column, substitution in registers), and the
// inverses of 32, 64 and 128 rows follow in place from
//     [[L11, 0], [L21, L22]]^-1 = [[X11, 0], [-X22 L21 X11, X22]],
// two DMMA products per doubling that skip the zero halves of X11 and X22.  The result, with
// zeros in the opposite triangle (what rocblas_trtri_fill does, rocblas_trtri.hpp:393-426), is
// written to invA.  FP32 blocks are inverted in FP64 and rounded once.
//
// The kernel is a chain of short steps (a solve waits for it before its first block), so it is
// bound by latency: copies that are all in flight at once, seven CTA barriers, and no index
// arithmetic beyond constants: 14 us for up to 148 FP64 blocks of 128 (FP32 16) where the version on
// 32 x 32 tiles with computed tile indexes took 42 us (a third of a 512 x 256 solve).
//
// Diagonal semantics follow rocblas_custom_trtri_device (rocblas_trtri.hpp:128-141):
// diag == unit reads no diagonal and uses 1; a zero non-unit diagonal entry is treated as 1.
#pragma once
#include <type_traits>

#include "common.cuh"
#include "mbarrier.cuh"
#include "mma_f64.cuh"

namespace rb200
{

template <typename T>
struct TrtriParams
{
    int         k;            // order of A (the blocks tile A's diagonal)
    int         nb;           // block order (<= 128)
    BatchPtr<T> A;            // A(0,0) of every batch entry
    int64_t     lda;
    BatchPtr<T> inv;          // block b of batch entry e goes to inv.get(e) + b * inv_block_stride
    int64_t     ldinv;
    int64_t     inv_block_stride;
    int         upper, unit;
    int         batch_base;
    // variable batch: order and leading dimension per entry (A and inv then come from
    // pointer arrays); blocks beyond an entry's order exit at once
    const int*     vk   = nullptr;
    const int64_t* vlda = nullptr;
    // the alpha of the solve that the inverses are for: with 0 it reads neither them nor A, which
    // need not exist then, so nothing is done
    Scalar<T> alpha;
};

constexpr int kTrtriNB      = 128;
constexpr int kTrtriThreads = 256; // 8 warps
// Column pitch in shared memory (column-major): the fragment reads, lanes (g, t) at element (g, t)
// or (t, g), are free of bank conflicts with a pitch of 4 mod 16 doubles.
constexpr int kTrtriLd  = kTrtriNB + 4;
constexpr int kTrtriLdT = kTrtriNB / 2 + 4; // temporary of at most 64 x 64

template <typename T>
constexpr size_t trtri_smem_bytes()
{
    return sizeof(double) * (size_t)(kTrtriNB * kTrtriLd + kTrtriNB / 2 * kTrtriLdT);
}

// NT neighbouring 16 x 8 tiles acc[n] += P(r0.., k) Q(k, c0 + 8n ..) over k in [k0, k1); P and Q
// column-major with pitches ldp, ldq.
template <int NT>
__device__ __forceinline__ void trtri_mma(double (&acc)[NT][4], const double* P, int ldp, const double* Q, int ldq,
                                          int k0, int k1, int g, int t)
{
#pragma unroll 2
    for(int k = k0; k < k1; k += 8)
    {
        const double* a0 = P + (k + t) * ldp + g;
        const double* a1 = P + (k + t + 4) * ldp + g;
        const double  a[4] = {a0[0], a0[8], a1[0], a1[8]};
#pragma unroll
        for(int n = 0; n < NT; ++n)
        {
            const double* q    = Q + (8 * n + g) * ldq + k + t;
            const double  b[2] = {q[0], q[4]};
            dmma_16x8x8(acc[n], a, b);
        }
    }
}

// The inverse of the lower triangular 128 x 128 block at X (column-major, pitch kTrtriLd, zero above
// the diagonal), in place, by 256 threads between two CTA barriers (the caller's before it, the
// last of its own after it).  Tm: 64 columns of kTrtriLdT doubles.  Returns (in all threads) whether
// everything it wrote is finite: if not, the zeros of a triangle may have met an infinity or NaN in a
// product, and rows may not be finite that do not depend on it; trtri_invert_rows is for that case.
__device__ __forceinline__ bool trtri_invert(double* X, double* Tm, bool zero_is_one)
{
    bool finite = true;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    // ---- 16 x 16 diagonal tiles: warp w inverts tile w, lane = column ----------------------------
    {
        constexpr int S = 16;
        double* const D = X + warp * S * (kTrtriLd + 1);
        double        d = lane < S ? D[lane * (kTrtriLd + 1)] : 1.0;
        if(zero_is_one && d == 0.0)
            d = 1.0;
        const double rd = 1.0 / d;
        double       x[S];
#pragma unroll
        for(int i = 0; i < S; ++i)
            x[i] = i == lane ? 1.0 : 0.0;
#pragma unroll
        for(int c = 0; c < S; ++c)
        {
            x[c] *= __shfl_sync(0xffffffffu, rd, c);
#pragma unroll
            for(int i = c + 1; i < S; ++i)
                x[i] -= D[c * kTrtriLd + i] * x[c];
        }
        __syncwarp();
        if(lane < S)
#pragma unroll
            for(int i = 0; i < S; ++i)
            {
                finite                 = finite && (i < lane || is_finite(x[i]));
                D[lane * kTrtriLd + i] = x[i];
            }
    }
    __syncthreads();

    // ---- 16 -> 32 -> 64 -> 128 ----------------------------------------------------------------
    // Of a doubling from S, the warp takes NT tiles of 16 x 8 at row rb, column cb of pair pr.
    auto doubling = [&](auto s_const, auto nt_const, int pr, int rb, int cb) {
        constexpr int S = decltype(s_const)::value, NT = decltype(nt_const)::value;
        double* const X11 = X + pr * 2 * S * (kTrtriLd + 1);
        double* const L21 = X11 + S;
        double* const X22 = X11 + S * (kTrtriLd + 1);
        double* const Tp  = Tm + pr * S * kTrtriLdT; // its S columns of the temporary
        double        acc[NT][4] = {};
        // Tp = L21 X11: X11's column c is zero above row c
        trtri_mma<NT>(acc, L21 + rb, kTrtriLd, X11 + cb * kTrtriLd, kTrtriLd, cb, S, g, t);
#pragma unroll
        for(int n = 0; n < NT; ++n)
#pragma unroll
            for(int e = 0; e < 4; ++e)
            {
                Tp[(cb + 8 * n + 2 * t + (e & 1)) * kTrtriLdT + rb + g + (e >> 1) * 8] = acc[n][e];
                acc[n][e] = 0.0;
            }
        __syncthreads();
        // X21 = -X22 Tp, over L21: X22's row r ends at column r
        trtri_mma<NT>(acc, X22 + rb, kTrtriLd, Tp + cb * kTrtriLdT, kTrtriLdT, 0, rb + 16, g, t);
#pragma unroll
        for(int n = 0; n < NT; ++n)
#pragma unroll
            for(int e = 0; e < 4; ++e)
            {
                finite = finite && is_finite(acc[n][e]);
                L21[(cb + 8 * n + 2 * t + (e & 1)) * kTrtriLd + rb + g + (e >> 1) * 8] = -acc[n][e];
            }
        if(S < kTrtriNB / 2)
            __syncthreads();
    };
    doubling(std::integral_constant<int, 16>{}, std::integral_constant<int, 1>{}, warp >> 1, 0, (warp & 1) * 8);
    doubling(std::integral_constant<int, 32>{}, std::integral_constant<int, 2>{}, warp >> 2, (warp & 1) * 16,
             (warp & 2) * 8);
    // warps w and w + 4 share a scheduler: opposite row blocks give it even work in both products
    doubling(std::integral_constant<int, 64>{}, std::integral_constant<int, 4>{}, 0,
             (warp < 4 ? warp : 7 - warp) * 16, (warp >> 2) * 32);
    return __syncthreads_and(finite) != 0;
}

// The inverse at X again, of the triangle L0[i di + j dj] (j <= i < n; the identity past n), with
// products over the triangles alone, so that what is not finite stays in the rows from its own on, as
// in a substitution: column after column from the last one, X21 = -X22 l21 / l11, thread = row.  About
// 0.1 ms; a function of its own, because the kernels around it are one pass through straight code and
// this inside them cost 2 us.
template <typename T>
__device__ __noinline__ void trtri_invert_rows(double* X, const T* L0, int64_t di, int64_t dj, int n, bool unit,
                                               bool zero_is_one)
{
    const int r = threadIdx.x;
    for(int e = r; e < kTrtriNB * kTrtriNB; e += kTrtriThreads)
    {
        const int i = e % kTrtriNB, j = e / kTrtriNB;
        double    v = 0.0;
        if(j < i && i < n)
            v = (double)L0[i * di + j * dj];
        else if(i == j)
        {
            v = i < n && !unit ? (double)L0[i * (di + dj)] : 1.0;
            if(zero_is_one && v == 0.0)
                v = 1.0;
        }
        X[j * kTrtriLd + i] = v;
    }
    __syncthreads();
    for(int c = kTrtriNB - 1; c >= 0; --c)
    {
        const double* const l  = X + c * kTrtriLd;
        const double        rd = 1.0 / l[c];
        double              v  = 0.0;
        if(r > c && r < kTrtriNB)
        {
            for(int k = c + 1; k <= r; ++k)
                v += X[k * kTrtriLd + r] * l[k];
            v = -v * rd;
        }
        __syncthreads();
        if(r >= c && r < kTrtriNB)
            X[c * kTrtriLd + r] = r == c ? rd : v;
        __syncthreads();
    }
}

template <typename T>
__global__ void __launch_bounds__(kTrtriThreads) trtri_block_kernel(TrtriParams<T> p)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* X  = reinterpret_cast<double*>(smem_raw); // the block, then its inverse in place
    double* Tm = X + kTrtriNB * kTrtriLd;

    const int     tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if(p.alpha.get() == T(0))
        return;
    const int     blk   = blockIdx.x;
    const int     batch = p.batch_base + blockIdx.y;
    const int     k     = p.vk ? p.vk[batch] : p.k;
    const int64_t lda   = p.vk ? p.vlda[batch] : p.lda;
    const int     r0    = blk * p.nb;
    if(r0 >= k)
        return; // (variable batch) this entry has fewer blocks
    const int bs = min(p.nb, k - r0);

    const T* A   = p.A.get(batch) + r0 + (int64_t)r0 * lda;
    T*       out = p.inv.get(batch) + (int64_t)blk * p.inv_block_stride;
    // (i, j) of the lower orientation is A(i, j), or A(bs - 1 - i, bs - 1 - j) of an upper block
    const T* const A0 = p.upper ? A + (int64_t)(bs - 1) * (lda + 1) : A;
    const int      sg = p.upper ? -1 : 1;

    // ---- stage the lower triangle, identity-padded to 128 -----------------------------------
    // Warp w takes the columns w, w + 8, ..; whole 32-row groups above the diagonal are left out.
    auto source = [&](int i, int j, bool& take) {
        take = i < bs && j < bs && (j < i || (i == j && !p.unit));
        return take ? A0 + sg * (i + (int64_t)j * lda) : A0;
    };
    if constexpr(std::is_same<T, double>::value)
    {
#pragma unroll
        for(int c = 0; c < kTrtriNB / 8; ++c)
#pragma unroll
            for(int u = c / 4; u < kTrtriNB / 32; ++u)
            {
                const int i = u * 32 + lane, j = c * 8 + warp;
                bool      take;
                const T*  src = source(i, j, take);
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_u32(X + j * kTrtriLd + i)),
                             "l"(src), "r"(take ? 8 : 0)
                             : "memory");
            }
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    else
    {
        // converted on the way: a row group's loads are all issued before its stores
#pragma unroll
        for(int u = 0; u < kTrtriNB / 32; ++u)
        {
            T v[4 * (kTrtriNB / 32)];
#pragma unroll
            for(int c = 0; c < 4 * (u + 1); ++c)
            {
                bool     take;
                const T* src = source(u * 32 + lane, c * 8 + warp, take);
                v[c]         = take ? *src : T(0);
            }
#pragma unroll
            for(int c = 0; c < 4 * (u + 1); ++c)
                X[(c * 8 + warp) * kTrtriLd + u * 32 + lane] = (double)v[c];
        }
    }
    __syncthreads();

    // unit diagonals and padding are staged as 0, which like a zero diagonal entry is read as 1
    if(!trtri_invert(X, Tm, true))
        trtri_invert_rows<T>(X, A0, sg, sg * lda, bs, p.unit, true);

    // ---- write inv(A_block) (bs x bs, ld = ldinv), zeros in the opposite triangle ----
    T* const out0 = p.upper ? out + (int64_t)(bs - 1) * (p.ldinv + 1) : out;
#pragma unroll 4
    for(int j = warp; j < bs; j += 8)
#pragma unroll
        for(int u = 0; u < kTrtriNB / 32; ++u)
        {
            const int i = u * 32 + lane;
            if(i < bs)
                out0[sg * (i + (int64_t)j * p.ldinv)] = i >= j ? (T)X[j * kTrtriLd + i] : T(0);
        }
}

} // namespace rb200

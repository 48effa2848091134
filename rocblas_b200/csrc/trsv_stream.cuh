// Triangular solve of one real right-hand side, op(A) x = b (rocblas_?trsv), as one read of A's
// triangle.  trsv_flag.cuh describes the scheme, the index map and the wait bounds, and serves
// several right-hand sides and callers whose workspace is too small for this kernel's exchange
// buffer.
//
// Below n ~ 30000 the time is not the triangle's bytes but the chain of 128-row blocks: what passes
// between one block's x and the next one's.  So here
//   * x travels as {value, 1} pairs that are written and polled as single 16-byte (FP32: 8-byte)
//     accesses: the poll that sees the tag has the value, with no fence before a flag and no second
//     round trip after it;
//   * a tile is streamed as two halves of 64 columns that alternate between two register buffers,
//     so the next half's loads are always in flight, and the whole tile next to the diagonal is in
//     registers before its x arrives;
//   * the diagonal block's inverse (trtri_invert) is built before the first wait, and x_b = inv y
//     uses every warp, 16 rows each, two lanes per row;
//   * blocks are claimed from a counter in order, so a block only ever waits for blocks whose CTAs
//     run.
// Measured (one B200, lower no-trans, against the flag solve): FP64 n = 256 85 -> 29 us, 4096 212 ->
// 80 us, 16384 733 -> 297 us (3.6 TB/s), 32768 1538 -> 797 us (5.4 TB/s); FP32 16384 656 -> 260 us.
// A block's hand-off takes 2.1 us, of which the poll is about half.
#pragma once
#include "trsv_flag.cuh"
#include "trtri_block.cuh"

namespace rb200
{

constexpr int kTsNB      = 128; // block rows
constexpr int kTsThreads = 256;

template <typename T>
constexpr size_t trsv_stream_exchange_bytes(int n)
{
    return 2 * sizeof(T) * (size_t)n;
}
// exchange pairs, then the claim counter
template <typename T>
constexpr size_t trsv_stream_workspace_bytes(int n)
{
    return trsv_stream_exchange_bytes<T>(n) + 16;
}
constexpr size_t trsv_stream_smem_bytes()
{
    return trtri_smem_bytes<double>();
}

__device__ __forceinline__ void ts_put(double* pair, double v)
{
    asm volatile("{\n\t.reg .b128 q;\n\tmov.b128 q, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], q;\n\t}" ::"l"(pair),
                 "l"(__double_as_longlong(v)), "l"(1ll)
                 : "memory");
}
__device__ __forceinline__ bool ts_get(const double* pair, double& v)
{
    long long lo, hi;
    asm volatile("{\n\t.reg .b128 q;\n\tld.relaxed.gpu.global.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
                 : "=l"(lo), "=l"(hi)
                 : "l"(pair)
                 : "memory");
    v = __longlong_as_double(lo);
    return hi != 0;
}
__device__ __forceinline__ void ts_put(float* pair, float v)
{
    const unsigned long long q = (1ull << 32) | __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(pair), "l"(q) : "memory");
}
__device__ __forceinline__ bool ts_get(const float* pair, float& v)
{
    unsigned long long q;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(q) : "l"(pair) : "memory");
    v = __uint_as_float((unsigned)q);
    return (q >> 32) != 0;
}

// TR: op(A) = A^T.  xch: trsv_stream_workspace_bytes, zero on entry; p.flags is not used.
template <typename T, bool TR>
__global__ void __launch_bounds__(kTsThreads, 1) trsv_stream_kernel(const TrsvParams<T> p, T* xch)
{
    constexpr int NV = 32; // elements of a half tile per lane
    extern __shared__ __align__(16) unsigned char ts_smem[];
    double* const X    = reinterpret_cast<double*>(ts_smem); // the diagonal block, then its inverse
    double* const Tm   = X + kTrtriNB * kTrtriLd;            // scratch of the inversion, then:
    double* const part = Tm;                                 // the warps' partial sums [warp][row] and
    double* const y    = Tm + kTsThreads / 32 * kTsNB;       // b - sum
    __shared__ int s_blk, s_stop;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nblk = (p.n + kTsNB - 1) / kTsNB;
    int* const counter = reinterpret_cast<int*>(xch + 2 * (size_t)p.n);
    // M(i, j) in logical indices: M0[i sI + j sJ]
    const int64_t  sgn = p.rev ? -1 : 1;
    const int64_t  sI = sgn * (TR ? p.lda : 1), sJ = sgn * (TR ? 1 : p.lda);
    const T* const M0 = p.A + (p.rev ? (int64_t)(p.n - 1) * (p.lda + 1) : 0);
    if(tid == 0)
        s_stop = 0;
    for(;;)
    {
        __syncthreads();
        if(tid == 0)
            s_blk = atomicAdd(counter, 1);
        __syncthreads();
        const int b = s_blk;
        if(b >= nblk)
            break;
        const int r0 = b * kTsNB, rows = min(kTsNB, p.n - r0);

        // ---- the diagonal block (identity past the matrix), inverted before any wait --------------
        for(int e = warp; e < kTsNB; e += kTsThreads / 32)
#pragma unroll
            for(int u = 0; u < kTsNB / 32; ++u)
            {
                const int  f = u * 32 + lane;
                const int  i = TR ? e : f, j = TR ? f : e; // lanes along A's contiguous direction
                double     v = 0.0;
                const bool one = i == j && (p.unit || i >= rows);
                if(j <= i && i < rows && !one)
                    v = (double)M0[(r0 + i) * sI + (r0 + j) * sJ];
                X[j * kTrtriLd + i] = one ? 1.0 : v;
            }
        __syncthreads();
        if(!trtri_invert(X, Tm, false))
            trtri_invert_rows<T>(X, M0 + r0 * (sI + sJ), sI, sJ, rows, p.unit, false);

        // ---- the tiles left of it, in halves of 64 columns ----------------------------------------
        // no-trans: lane = 4 rows, warp = 8 columns; trans: lane = 2 columns, warp = 16 rows
        T          buf0[NV], buf1[NV];
        constexpr int NACC = TR ? 16 : 4;
        T          acc[NACC];
#pragma unroll
        for(int q = 0; q < NACC; ++q)
            acc[q] = T(0);
        const T* const tile = M0 + (TR ? (int64_t)(r0 + warp * 16) * sI + lane * sJ
                                       : (int64_t)(r0 + lane) * sI + warp * 8 * sJ);
        auto load = [&](T (&v)[NV], int h) {
            const T* src = tile + (int64_t)h * 64 * sJ;
            if(TR)
            {
#pragma unroll
                for(int q = 0; q < 16; ++q, src += sI)
#pragma unroll
                    for(int u = 0; u < 2; ++u)
                        v[2 * q + u] = warp * 16 + q < rows ? src[u * 32 * sJ] : T(0);
            }
            else
            {
#pragma unroll
                for(int q = 0; q < 8; ++q, src += sJ)
#pragma unroll
                    for(int u = 0; u < 4; ++u)
                        v[4 * q + u] = lane + 32 * u < rows ? src[u * 32 * sI] : T(0);
            }
        };
        // this lane's x of block j, both halves at once: no-trans lanes 0..7 hold the warp's 8 columns
        // of the first half and lanes 8..15 those of the second, trans every lane 4 columns
        constexpr int NX = TR ? 4 : 1;
        struct Xv
        {
            T    v[NX];
            bool ok;
        };
        const T* const xsrc = xch + 2 * (TR ? lane : (lane & 8) * 8 + warp * 8 + (lane & 7));
        auto fetch = [&](int j, Xv& x) {
            x.ok = true;
#pragma unroll
            for(int u = 0; u < NX; ++u)
                x.ok = ts_get(xsrc + 2 * ((int64_t)j * kTsNB + 32 * u), x.v[u]) && x.ok;
        };
        auto await = [&](int j, Xv& x) {
            if(__all_sync(0xffffffffu, x.ok))
                return;
            const long long t0 = clock64();
            do
            {
                if(*(volatile int*)&s_stop || clock64() - t0 > p.wait_cycles)
                {
                    atomicCAS(p.error, 0, 5);
                    *(volatile int*)&s_stop = 1;
                    break;
                }
                fetch(j, x);
            } while(!x.ok);
            __syncwarp();
        };
        auto add = [&](const T (&v)[NV], const Xv& x, auto half) {
            constexpr int H = decltype(half)::value;
            if(TR)
            {
#pragma unroll
                for(int q = 0; q < NACC; ++q)
                    acc[q] += v[2 * q] * x.v[(2 * H) % NX] + v[2 * q + 1] * x.v[(2 * H + 1) % NX];
            }
            else
            {
#pragma unroll
                for(int q = 0; q < 8; ++q)
                {
                    const T xv = __shfl_sync(0xffffffffu, x.v[0], 8 * H + q);
#pragma unroll
                    for(int u = 0; u < 4; ++u)
                        acc[u] += v[4 * q + u] * xv;
                }
            }
        };
        // b's entry, read before any wait (no other block writes it); thread = row
        const double bv = tid < rows ? (double)*tv_x(p, r0 + tid) : 0.0;
        Xv x, xn;
        if(b > 0)
        {
            load(buf0, 0);
            fetch(0, x);
        }
#pragma unroll 1
        for(int j = 0; j < b; ++j)
        {
            load(buf1, 2 * j + 1);
            await(j, x);
            add(buf0, x, std::integral_constant<int, 0>{});
            if(j + 1 < b)
            {
                load(buf0, 2 * j + 2);
                fetch(j + 1, xn);
            }
            add(buf1, x, std::integral_constant<int, 1>{});
            x = xn;
        }

        // ---- y = b - sum ---------------------------------------------------------------------------
        if(TR)
        {
            // 16 rows over 32 lanes: halve the rows a lane holds at each exchange; row = lane / 2
#pragma unroll
            for(int w = 16, m = 8; m >= 1; w >>= 1, m >>= 1)
#pragma unroll
                for(int q = 0; q < 8; ++q)
                    if(q < m)
                    {
                        const bool up   = (lane & w) != 0;
                        const T    mine = up ? acc[(q + m) % NACC] : acc[q % NACC];
                        const T    give = up ? acc[q % NACC] : acc[(q + m) % NACC];
                        acc[q % NACC]   = mine + __shfl_xor_sync(0xffffffffu, give, w);
                    }
            acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
            if(!(lane & 1))
                part[warp * 16 + (lane >> 1)] = (double)acc[0];
        }
        else
        {
#pragma unroll
            for(int u = 0; u < 4; ++u)
                part[warp * kTsNB + lane + 32 * u] = (double)acc[u % NACC];
        }
        __syncthreads();
        if(tid < kTsNB)
        {
            double s;
            if(TR)
                s = part[tid];
            else
            {
                double v[kTsThreads / 32];
#pragma unroll
                for(int w = 0; w < kTsThreads / 32; ++w)
                    v[w] = part[w * kTsNB + tid];
                s = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
            }
            y[tid] = bv - s;
        }
        if(__syncthreads_or(*(volatile int*)&s_stop))
            break;

        // ---- x_b = inv y: warp = 16 rows, the lane pair (l, l + 16) the even and odd columns ---------
        {
            const int     row = warp * 16 + (lane & 15), c0 = lane >> 4;
            const double* xr  = X + row;
            double        s[4] = {0.0, 0.0, 0.0, 0.0};
            for(int c = c0; c < warp * 16; c += 8)
#pragma unroll
                for(int u = 0; u < 4; ++u)
                    s[u] += xr[(c + 2 * u) * kTrtriLd] * y[c + 2 * u];
            // the diagonal tile: columns past the row must not reach it, whatever y holds
#pragma unroll
            for(int u = 0; u < 8; ++u)
            {
                const int c = warp * 16 + c0 + 2 * u;
                if(c <= row)
                    s[u & 3] += xr[c * kTrtriLd] * y[c];
            }
            double v = (s[0] + s[1]) + (s[2] + s[3]);
            v += __shfl_xor_sync(0xffffffffu, v, 16);
            if(lane < 16 && row < rows)
            {
                ts_put(xch + 2 * (size_t)(r0 + row), (T)v);
                *tv_x(p, r0 + row) = (T)v;
            }
        }
    }
}

} // namespace rb200

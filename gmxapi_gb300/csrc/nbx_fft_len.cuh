// Axis passes of the PME transforms for lengths n = R1 R2 known at compile time.
//
// A line takes max(R1, R2) threads.  Thread j < R2 loads the points j + R2 r (r < R1) into
// registers, does their R1-point DFT, multiplies output q by exp(-+ 2 pi i j q / n) and puts it in
// shared memory; thread q < R1 then reads the R2 values of its q and their R2-point DFT gives the
// points q + R1 s in natural order.  One trip through shared memory per line instead of one per
// radix-4/2/3/5 stage: the passes are bound by latency (the grids sit in L2), and a thread has all
// its loads in flight at once.  96^3 / 120^3 grids, per pass: 7.5 / 8.4 us with a warp per line and
// four or five Stockham stages, 4.6-5.0 / 5.7-6.8 us now (the x pass with the solve 7.6, with energies
// 11.3 us at 120^3).
//
// The strided passes (y and x) take kCols consecutive z-frequencies of a line per block, thread
// (j, c) with c fastest, so global rows of 64 bytes are read and written whole, without staging.
#pragma once

#include "nbx_internal.cuh"
#include "nbx_fft.cuh"
#include "nbx_pme_solve.cuh"

#include <type_traits>

namespace nbx
{

namespace fftr
{

// cos and sin of 2 pi k / n in double, for k >= 0, from their Maclaurin series after reduction to
// [-pi, pi] (26 terms: the first dropped is below 1e-26)
__host__ __device__ constexpr double turn(int k, int n)
{
    const int r = k % n;
    return 6.283185307179586476925 * (2 * r > n ? (double)(r - n) : (double)r) / (double)n;
}
__host__ __device__ constexpr double cos_turn(int k, int n)
{
    const double x = turn(k, n);
    double       t = 1.0, s = 1.0;
    for (int i = 1; i < 26; i++)
    {
        t *= -x * x / ((2.0 * i - 1.0) * (2.0 * i));
        s += t;
    }
    return s;
}
__host__ __device__ constexpr double sin_turn(int k, int n)
{
    const double x = turn(k, n);
    double       t = x, s = x;
    for (int i = 1; i < 26; i++)
    {
        t *= -x * x / ((2.0 * i) * (2.0 * i + 1.0));
        s += t;
    }
    return s;
}

__device__ __forceinline__ float2 add(float2 a, float2 b)
{
    return make_float2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ float2 sub(float2 a, float2 b)
{
    return make_float2(a.x - b.x, a.y - b.y);
}

// v exp(-+ 2 pi i K / R), K and R known at compile time
template<int K, int R, bool kInv>
__device__ __forceinline__ float2 rotate(float2 v)
{
    constexpr int k = K % R;
    if constexpr (k == 0)
    {
        return v;
    }
    else if constexpr (2 * k == R)
    {
        return make_float2(-v.x, -v.y);
    }
    else if constexpr (4 * k == R || 4 * k == 3 * R)
    {
        // -i forward for a quarter turn, +i for three quarters (and the other way round backward)
        return ((4 * k == R) != kInv) ? make_float2(v.y, -v.x) : make_float2(-v.y, v.x);
    }
    else
    {
        constexpr float c = (float)cos_turn(k, R);
        constexpr float s = (float)(kInv ? sin_turn(k, R) : -sin_turn(k, R));
        return make_float2(fmaf(v.x, c, -v.y * s), fmaf(v.x, s, v.y * c));
    }
}

template<int I, int N, class F>
__device__ __forceinline__ void each(const F& f)
{
    if constexpr (I < N)
    {
        f(std::integral_constant<int, I>{});
        each<I + 1, N>(f);
    }
}

__host__ __device__ constexpr int first_factor(int r)
{
    return r == 4 ? 2 : r % 4 == 0 ? 4 : r % 2 == 0 ? 2 : r % 3 == 0 ? 3 : r % 5 == 0 ? 5 : r;
}

// R-point DFT in registers, V_q = sum_r v_r exp(-+ 2 pi i q r / R), natural order.  Composite R as
// A x B (A sub-transforms' outputs rotated by constants), odd primes from the sums and differences
// v_k +- v_{R-k}.
template<int R, bool kInv>
__device__ __forceinline__ void dft(float2 (&v)[R])
{
    constexpr int A = first_factor(R);
    if constexpr (R == 1)
    {
        return;
    }
    else if constexpr (R == 2)
    {
        const float2 a = v[0], b = v[1];
        v[0]           = add(a, b);
        v[1]           = sub(a, b);
    }
    else if constexpr (A == R)
    {
        constexpr int H = (R - 1) / 2;
        float2        t[H], u[H];
        const float2  v0 = v[0];
        each<0, H>([&](auto K) {
            constexpr int k = decltype(K)::value;
            t[k]            = add(v[k + 1], v[R - 1 - k]);
            u[k]            = sub(v[k + 1], v[R - 1 - k]);
            v[0]            = add(v[0], t[k]);
        });
        each<1, H + 1>([&](auto Q) {
            constexpr int q = decltype(Q)::value;
            float2        a = v0, b = make_float2(0.0f, 0.0f);
            each<0, H>([&](auto K) {
                constexpr int   k = decltype(K)::value;
                constexpr float c = (float)cos_turn(q * (k + 1), R), s = (float)sin_turn(q * (k + 1), R);
                a                 = make_float2(fmaf(c, t[k].x, a.x), fmaf(c, t[k].y, a.y));
                b                 = make_float2(fmaf(s, u[k].x, b.x), fmaf(s, u[k].y, b.y));
            });
            // forward: V_q = a - i b, V_{R-q} = a + i b
            const float2 m = make_float2(a.x + b.y, a.y - b.x), p = make_float2(a.x - b.y, a.y + b.x);
            v[q]     = kInv ? p : m;
            v[R - q] = kInv ? m : p;
        });
    }
    else
    {
        constexpr int B = R / A;
        float2        y[R];  // [q][b]
        each<0, B>([&](auto Bi) {
            constexpr int b = decltype(Bi)::value;
            float2        w[A];
            each<0, A>([&](auto Ai) {
                constexpr int a = decltype(Ai)::value;
                w[a]            = v[b + B * a];
            });
            dft<A, kInv>(w);
            each<0, A>([&](auto Q) {
                constexpr int q = decltype(Q)::value;
                y[q * B + b]    = rotate<b * q, R, kInv>(w[q]);
            });
        });
        each<0, A>([&](auto Q) {
            constexpr int q = decltype(Q)::value;
            float2        w[B];
            each<0, B>([&](auto Bi) {
                constexpr int b = decltype(Bi)::value;
                w[b]            = y[q * B + b];
            });
            dft<B, kInv>(w);
            each<0, B>([&](auto S) {
                constexpr int s = decltype(S)::value;
                v[q + A * s]    = w[s];
            });
        });
    }
}

// v[q] *= exp(-+ 2 pi i j q / n), q > 0, from the root table in global memory (j q < n)
template<int R, bool kInv>
__device__ __forceinline__ void twiddle(float2 (&v)[R], const float2* __restrict__ roots, int j)
{
    float2 w[R];
#pragma unroll
    for (int q = 1; q < R; q++)
    {
        w[q] = __ldg(&roots[j * q]);
    }
#pragma unroll
    for (int q = 1; q < R; q++)
    {
        v[q] = cmul(v[q], kInv ? make_float2(w[q].x, -w[q].y) : w[q]);
    }
}

constexpr int round32(int n)
{
    return (n + 31) / 32 * 32;
}

template<int R1, int R2>
struct Shape
{
    static constexpr int n       = R1 * R2;
    static constexpr int threads = R1 > R2 ? R1 : R2;  // per line
    static constexpr int row     = R2 | 1;             // exchange rows of odd length: no bank conflicts
};

constexpr int kZPairs = 8;  // line pairs per block of the z passes
constexpr int kCols   = 8;  // z-frequencies per block of the strided passes

// z forward: lines 2p and 2p + 1 of the real grid as one complex line a + i b, then
// A_k = (Z_k + conj Z_{n-k}) / 2 and B_k = (Z_k - conj Z_{n-k}) / 2i for k = 0 .. n/2.
template<int R1, int R2>
__global__ void __launch_bounds__(round32(kZPairs* Shape<R1, R2>::threads))
        k_z_r2c(const float2* __restrict__ roots, const float* real, float2* cplx, int nlines)
{
    pdl_begin();
    using S              = Shape<R1, R2>;
    constexpr int n      = S::n, nzc = n / 2 + 1;
    constexpr int kLine  = R1 * S::row;
    __shared__ float2 sm[kZPairs * kLine];
    const int         p  = threadIdx.x / S::threads, j = threadIdx.x - p * S::threads;
    const int         la = 2 * (blockIdx.x * kZPairs + p);
    const bool        on = p < kZPairs && la < nlines, hb = la + 1 < nlines;
    float2* const     ln = sm + p * kLine;
    if (on && j < R2)
    {
        const float* a = real + (size_t)la * n;
        float2       v[R1];
#pragma unroll
        for (int r = 0; r < R1; r++)
        {
            v[r] = make_float2(a[j + R2 * r], hb ? a[n + j + R2 * r] : 0.0f);
        }
        dft<R1, false>(v);
        twiddle<R1, false>(v, roots, j);
#pragma unroll
        for (int q = 0; q < R1; q++)
        {
            ln[q * S::row + j] = v[q];
        }
    }
    __syncthreads();
    float2 w[R2];
    if (on && j < R1)
    {
#pragma unroll
        for (int b = 0; b < R2; b++)
        {
            w[b] = ln[j * S::row + b];
        }
        dft<R2, false>(w);
    }
    __syncthreads();
    if (on && j < R1)
    {
#pragma unroll
        for (int s = 0; s < R2; s++)
        {
            ln[j + R1 * s] = w[s];
        }
    }
    __syncthreads();
    const int lines = min(2 * kZPairs, nlines - 2 * (int)blockIdx.x * kZPairs);
    float2*   out   = cplx + (size_t)2 * blockIdx.x * kZPairs * nzc;
    for (int i = threadIdx.x; i < lines * nzc; i += blockDim.x)
    {
        const int     l  = i / nzc, k = i - l * nzc;
        const float2* z  = sm + (l >> 1) * kLine;
        const float2  zk = z[k], zn = z[k == 0 ? 0 : n - k];
        out[i] = (l & 1) ? make_float2(0.5f * (zk.y + zn.y), 0.5f * (zn.x - zk.x))
                         : make_float2(0.5f * (zk.x + zn.x), 0.5f * (zk.y - zn.y));
    }
}

// z backward: Z = A + i B over the full line (A_{n-k} = conj A_k), transformed back; the real and
// imaginary parts are lines 2p and 2p + 1.  The imaginary parts of A_0 and B_0 (and of A_{n/2},
// B_{n/2} for even n) are dropped, as a complex-to-real transform that assumes a Hermitian line does.
template<int R1, int R2>
__global__ void __launch_bounds__(round32(kZPairs* Shape<R1, R2>::threads))
        k_z_c2r(const float2* __restrict__ roots, const float2* cplx, float* real, int nlines)
{
    pdl_begin();
    using S              = Shape<R1, R2>;
    constexpr int n      = S::n, nzc = n / 2 + 1;
    constexpr int kLine  = R1 * S::row;
    __shared__ float2 sm[kZPairs * kLine];
    const int         p  = threadIdx.x / S::threads, j = threadIdx.x - p * S::threads;
    const int         la = 2 * (blockIdx.x * kZPairs + p);
    const bool        on = p < kZPairs && la < nlines, hb = la + 1 < nlines;
    float2* const     ln = sm + p * kLine;
    if (on && j < R2)
    {
        const float2* a = cplx + (size_t)la * nzc;
        float2        A[R1], B[R1];
#pragma unroll
        for (int r = 0; r < R1; r++)
        {
            const int k  = j + R2 * r;
            const int kk = k < nzc ? k : n - k;
            A[r]         = a[kk];
            B[r]         = hb ? a[nzc + kk] : make_float2(0.0f, 0.0f);
        }
        float2 v[R1];
#pragma unroll
        for (int r = 0; r < R1; r++)
        {
            const int   k  = j + R2 * r;
            const float sg = k >= nzc ? -1.0f : (k == 0 || 2 * k == n) ? 0.0f : 1.0f;
            v[r]           = make_float2(A[r].x - sg * B[r].y, fmaf(sg, A[r].y, B[r].x));
        }
        dft<R1, true>(v);
        twiddle<R1, true>(v, roots, j);
#pragma unroll
        for (int q = 0; q < R1; q++)
        {
            ln[q * S::row + j] = v[q];
        }
    }
    __syncthreads();
    if (on && j < R1)
    {
        float2 w[R2];
#pragma unroll
        for (int b = 0; b < R2; b++)
        {
            w[b] = ln[j * S::row + b];
        }
        dft<R2, true>(w);
        float* a = real + (size_t)la * n;
#pragma unroll
        for (int s = 0; s < R2; s++)
        {
            a[j + R1 * s] = w[s].x;
            if (hb)
            {
                a[n + j + R1 * s] = w[s].y;
            }
        }
    }
}

// Lines along y or x of the half-complex grid: block (outer index o, tile t), the tile's columns
// z-frequencies t kCols .. t kCols + kCols - 1.
template<int R1, int R2, bool kInv>
__global__ void __launch_bounds__(round32(kCols* Shape<R1, R2>::threads))
        k_strided(const float2* __restrict__ roots, float2* data, int elem_stride, int outer_stride,
                  int ntiles, int nzc)
{
    pdl_begin();
    using S = Shape<R1, R2>;
    __shared__ float2 sm[R1 * S::row * kCols];
    const int         o = blockIdx.x / ntiles, t = blockIdx.x - o * ntiles;
    const int         j = threadIdx.x / kCols, c = threadIdx.x % kCols;
    const bool        on   = t * kCols + c < nzc;
    float2* const     line = data + (size_t)o * outer_stride + t * kCols + c;
    if (on && j < R2)
    {
        float2 v[R1];
#pragma unroll
        for (int r = 0; r < R1; r++)
        {
            v[r] = line[(size_t)(j + R2 * r) * elem_stride];
        }
        dft<R1, kInv>(v);
        twiddle<R1, kInv>(v, roots, j);
#pragma unroll
        for (int q = 0; q < R1; q++)
        {
            sm[(q * S::row + j) * kCols + c] = v[q];
        }
    }
    __syncthreads();
    if (on && j < R1)
    {
        float2 w[R2];
#pragma unroll
        for (int b = 0; b < R2; b++)
        {
            w[b] = sm[(j * S::row + b) * kCols + c];
        }
        dft<R2, kInv>(w);
#pragma unroll
        for (int s = 0; s < R2; s++)
        {
            line[(size_t)(j + R1 * s) * elem_stride] = w[s];
        }
    }
}

// The x transform of the forward FFT, the Coulomb solve and the x transform of the backward FFT in
// one pass over the half-complex grid: thread q has the points q + R1 s of its column after the
// forward transform, scales them in registers, and starts the backward transform with them.
template<int R1, int R2, bool kEnergy>
__global__ void __launch_bounds__(round32(kCols* Shape<R1, R2>::threads))
        k_x_solve(const float2* __restrict__ roots, float2* cgrid, PmeSolve ps, int ntiles)
{
    pdl_begin();
    using S = Shape<R1, R2>;
    __shared__ float2 sm[R1 * S::row * kCols];
    const int         nzc = ps.d.n[2] / 2 + 1;
    const int         ky = blockIdx.x / ntiles, t = blockIdx.x - ky * ntiles;
    const int         j = threadIdx.x / kCols, c = threadIdx.x % kCols;
    const int         kz   = t * kCols + c;
    const bool        on   = kz < nzc;
    const size_t      es   = (size_t)ps.d.n[1] * nzc;
    float2* const     line = cgrid + (size_t)ky * nzc + kz;
    float             acc[7] = { 0, 0, 0, 0, 0, 0, 0 };
    if (on && j < R2)
    {
        float2 v[R1];
#pragma unroll
        for (int r = 0; r < R1; r++)
        {
            v[r] = line[(size_t)(j + R2 * r) * es];
        }
        dft<R1, false>(v);
        twiddle<R1, false>(v, roots, j);
#pragma unroll
        for (int q = 0; q < R1; q++)
        {
            sm[(q * S::row + j) * kCols + c] = v[q];
        }
    }
    __syncthreads();
    float2 w[R2];
    if (on && j < R1)
    {
#pragma unroll
        for (int b = 0; b < R2; b++)
        {
            w[b] = sm[(j * S::row + b) * kCols + c];
        }
        dft<R2, false>(w);
#pragma unroll
        for (int s = 0; s < R2; s++)
        {
            const int kx = j + R1 * s;
            if (kx != 0 || ky != 0 || kz != 0)
            {
                solve_point(ps.d, ps.bsp, ps.elfac, ps.factor, ps.pivol, kx, ky, kz, kEnergy, w[s], acc);
            }
        }
    }
    // the energy sums end here, under the other warps' transforms, and not with the kernel: 120^3 15.6 -> 11.3 us
    __shared__ double red[kEnergy ? 7 : 1][8];
    if (kEnergy)
    {
        solve_add_warp(acc, red);
    }
    if (on && j < R1)
    {
        dft<R2, true>(w);
        twiddle<R2, true>(w, roots, j);
    }
    __syncthreads();
    if (kEnergy)
    {
        solve_add_block(red, ps.partials);
    }
    if (on && j < R1)
    {
#pragma unroll
        for (int b = 0; b < R2; b++)
        {
            sm[(j * S::row + b) * kCols + c] = w[b];
        }
    }
    __syncthreads();
    if (on && j < R2)
    {
        float2 v[R1];
#pragma unroll
        for (int q = 0; q < R1; q++)
        {
            v[q] = sm[(q * S::row + j) * kCols + c];
        }
        dft<R1, true>(v);
#pragma unroll
        for (int r = 0; r < R1; r++)
        {
            line[(size_t)(j + R2 * r) * es] = v[r];
        }
    }
}

// ---- z and y in one kernel: a block per x plane of a grid with ny = nz ----
// The planes are small (96^2: 37 KB) and the passes bound by latency, so a plane stays in shared memory
// between the z and the y transforms: one kernel and one trip through L2 instead of two.  Thread (p, j)
// takes a line pair in the z part, thread (c, j) a column in the y part.  A convolution of 3 000 atoms
// went from 24.1 to 20.5 us, of 288 000 atoms (120^3) from 86.6 to 82.6 us, 20 steps of dynamics of
// 32 000 atoms from 1925 to 1836 us.  Taken up to 768 threads (n <= 120 but 112); longer lines need more
// threads than a block has or leave it fewer than 80 registers a thread, and keep a pass per axis.
template<int R1, int R2>
struct Plane
{
    using S                      = Shape<R1, R2>;
    static constexpr int n       = S::n;
    static constexpr int nzc     = n / 2 + 1;
    static constexpr int pairs   = (n + 1) / 2;
    static constexpr int line    = R1 * S::row;  // exchange words of one line
    static constexpr int threads = round32(nzc * S::threads);
    static constexpr int words   = nzc * line > n * nzc ? nzc * line : n * nzc;  // pairs <= nzc
    static constexpr bool fits   = threads <= 768;
};

template<int R1, int R2>
__global__ void __launch_bounds__(Plane<R1, R2>::threads)
        k_plane_r2c(const float2* __restrict__ roots, const float* real, float2* cplx)
{
    pdl_begin();
    using S = Shape<R1, R2>;
    using P = Plane<R1, R2>;
    constexpr int n = P::n, nzc = P::nzc;
    extern __shared__ float2 psm[];
    {
        const int     p  = threadIdx.x / S::threads, j = threadIdx.x - p * S::threads;
        const bool    on = p < P::pairs, hb = 2 * p + 1 < n;
        float2* const ln = psm + p * P::line;
        if (on && j < R2)
        {
            const float* a = real + ((size_t)blockIdx.x * n + 2 * p) * n;
            float2       v[R1];
#pragma unroll
            for (int r = 0; r < R1; r++)
            {
                v[r] = make_float2(a[j + R2 * r], hb ? a[n + j + R2 * r] : 0.0f);
            }
            dft<R1, false>(v);
            twiddle<R1, false>(v, roots, j);
#pragma unroll
            for (int q = 0; q < R1; q++)
            {
                ln[q * S::row + j] = v[q];
            }
        }
        __syncthreads();
        float2 w[R2];
        if (on && j < R1)
        {
#pragma unroll
            for (int b = 0; b < R2; b++)
            {
                w[b] = ln[j * S::row + b];
            }
            dft<R2, false>(w);
        }
        __syncthreads();
        if (on && j < R1)
        {
#pragma unroll
            for (int s = 0; s < R2; s++)
            {
                ln[j + R1 * s] = w[s];
            }
        }
        __syncthreads();
    }
    // column c (z-frequency) along y: the value of line y comes from the pair y / 2 (see k_z_r2c)
    const int  j = threadIdx.x / nzc, c = threadIdx.x - j * nzc;
    const bool in = j < R2, out = j < R1;
    float2     v[R1];
    if (in)
    {
#pragma unroll
        for (int r = 0; r < R1; r++)
        {
            const int     y  = j + R2 * r;
            const float2* z  = psm + (y >> 1) * P::line;
            const float2  zk = z[c], zn = z[c == 0 ? 0 : n - c];
            v[r] = (y & 1) ? make_float2(0.5f * (zk.y + zn.y), 0.5f * (zn.x - zk.x))
                           : make_float2(0.5f * (zk.x + zn.x), 0.5f * (zk.y - zn.y));
        }
        dft<R1, false>(v);
        twiddle<R1, false>(v, roots, j);
    }
    __syncthreads();
    if (in)
    {
#pragma unroll
        for (int q = 0; q < R1; q++)
        {
            psm[(q * S::row + j) * nzc + c] = v[q];
        }
    }
    __syncthreads();
    if (out)
    {
        float2 w[R2];
#pragma unroll
        for (int b = 0; b < R2; b++)
        {
            w[b] = psm[(j * S::row + b) * nzc + c];
        }
        dft<R2, false>(w);
        float2* o = cplx + (size_t)blockIdx.x * n * nzc + c;
#pragma unroll
        for (int s = 0; s < R2; s++)
        {
            o[(j + R1 * s) * nzc] = w[s];
        }
    }
}

template<int R1, int R2>
__global__ void __launch_bounds__(Plane<R1, R2>::threads)
        k_plane_c2r(const float2* __restrict__ roots, const float2* cplx, float* real)
{
    pdl_begin();
    using S = Shape<R1, R2>;
    using P = Plane<R1, R2>;
    constexpr int n = P::n, nzc = P::nzc;
    extern __shared__ float2 psm[];
    {
        const int  j = threadIdx.x / nzc, c = threadIdx.x - j * nzc;
        const bool in = j < R2, out = j < R1;
        if (in)
        {
            const float2* a = cplx + (size_t)blockIdx.x * n * nzc + c;
            float2        v[R1];
#pragma unroll
            for (int r = 0; r < R1; r++)
            {
                v[r] = a[(j + R2 * r) * nzc];
            }
            dft<R1, true>(v);
            twiddle<R1, true>(v, roots, j);
#pragma unroll
            for (int q = 0; q < R1; q++)
            {
                psm[(q * S::row + j) * nzc + c] = v[q];
            }
        }
        __syncthreads();
        float2 w[R2];
        if (out)
        {
#pragma unroll
            for (int b = 0; b < R2; b++)
            {
                w[b] = psm[(j * S::row + b) * nzc + c];
            }
            dft<R2, true>(w);
        }
        __syncthreads();
        if (out)
        {
#pragma unroll
            for (int s = 0; s < R2; s++)
            {
                psm[(j + R1 * s) * nzc + c] = w[s];
            }
        }
        __syncthreads();
    }
    // lines 2p and 2p + 1 along z (see k_z_c2r)
    const int  p  = threadIdx.x / S::threads, j = threadIdx.x - p * S::threads;
    const bool on = p < P::pairs, hb = 2 * p + 1 < n;
    float2     v[R1];
    if (on && j < R2)
    {
        const float2* a = psm + 2 * p * nzc;
#pragma unroll
        for (int r = 0; r < R1; r++)
        {
            const int    k  = j + R2 * r;
            const int    kk = k < nzc ? k : n - k;
            const float  sg = k >= nzc ? -1.0f : (k == 0 || 2 * k == n) ? 0.0f : 1.0f;
            const float2 A  = a[kk], B = hb ? a[nzc + kk] : make_float2(0.0f, 0.0f);
            v[r]            = make_float2(A.x - sg * B.y, fmaf(sg, A.y, B.x));
        }
        dft<R1, true>(v);
        twiddle<R1, true>(v, roots, j);
    }
    __syncthreads();
    float2* const ln = psm + p * P::line;
    if (on && j < R2)
    {
#pragma unroll
        for (int q = 0; q < R1; q++)
        {
            ln[q * S::row + j] = v[q];
        }
    }
    __syncthreads();
    if (on && j < R1)
    {
        float2 w[R2];
#pragma unroll
        for (int b = 0; b < R2; b++)
        {
            w[b] = ln[j * S::row + b];
        }
        dft<R2, true>(w);
        float* a = real + ((size_t)blockIdx.x * n + 2 * p) * n;
#pragma unroll
        for (int s = 0; s < R2; s++)
        {
            a[j + R1 * s] = w[s].x;
            if (hb)
            {
                a[n + j + R1 * s] = w[s].y;
            }
        }
    }
}

template<int R1, int R2>
cudaError_t launch_plane_r2c(const float2* roots, const float* real, float2* cplx, int nx, cudaStream_t s)
{
    constexpr size_t smem = sizeof(float2) * Plane<R1, R2>::words;
    cudaError_t      e    = smem_optin<k_plane_r2c<R1, R2>>(smem, smem);
    if (e == cudaSuccess)
    {
        e = launch_pdl(k_plane_r2c<R1, R2>, nx, Plane<R1, R2>::threads, smem, s, roots, real, cplx);
    }
    return e;
}

template<int R1, int R2>
cudaError_t launch_plane_c2r(const float2* roots, const float2* cplx, float* real, int nx, cudaStream_t s)
{
    constexpr size_t smem = sizeof(float2) * Plane<R1, R2>::words;
    cudaError_t      e    = smem_optin<k_plane_c2r<R1, R2>>(smem, smem);
    if (e == cudaSuccess)
    {
        e = launch_pdl(k_plane_c2r<R1, R2>, nx, Plane<R1, R2>::threads, smem, s, roots, cplx, real);
    }
    return e;
}

template<int R1, int R2>
void launch_z_r2c(const float2* roots, const float* real, float2* cplx, int nlines, cudaStream_t s)
{
    const int blocks = (nlines + 2 * kZPairs - 1) / (2 * kZPairs);
    launch_pdl(k_z_r2c<R1, R2>, blocks, round32(kZPairs * Shape<R1, R2>::threads), 0, s, roots, real, cplx, nlines);
}

template<int R1, int R2>
void launch_z_c2r(const float2* roots, const float2* cplx, float* real, int nlines, cudaStream_t s)
{
    const int blocks = (nlines + 2 * kZPairs - 1) / (2 * kZPairs);
    launch_pdl(k_z_c2r<R1, R2>, blocks, round32(kZPairs * Shape<R1, R2>::threads), 0, s, roots, cplx, real, nlines);
}

template<int R1, int R2>
void launch_strided(bool inv, const float2* roots, float2* data, int nouter, int elem, int outer, int nzc,
                    cudaStream_t s)
{
    const int ntiles = (nzc + kCols - 1) / kCols, threads = round32(kCols * Shape<R1, R2>::threads);
    if (inv)
    {
        launch_pdl(k_strided<R1, R2, true>, nouter * ntiles, threads, 0, s, roots, data, elem, outer, ntiles, nzc);
    }
    else
    {
        launch_pdl(k_strided<R1, R2, false>, nouter * ntiles, threads, 0, s, roots, data, elem, outer, ntiles, nzc);
    }
}

template<int R1, int R2>
void launch_x_solve(const float2* roots, float2* cgrid, const PmeSolve& ps, cudaStream_t s)
{
    const int ntiles = (ps.d.n[2] / 2 + 1 + kCols - 1) / kCols, threads = round32(kCols * Shape<R1, R2>::threads);
    if (ps.partials)
    {
        launch_pdl(k_x_solve<R1, R2, true>, ps.d.n[1] * ntiles, threads, 0, s, roots, cgrid, ps, ntiles);
    }
    else
    {
        launch_pdl(k_x_solve<R1, R2, false>, ps.d.n[1] * ntiles, threads, 0, s, roots, cgrid, ps, ntiles);
    }
}

template<int R1, int R2>
constexpr FftLen make_len()
{
    FftLen l = { R1 * R2, launch_z_r2c<R1, R2>, launch_z_c2r<R1, R2>, launch_strided<R1, R2>, launch_x_solve<R1, R2>,
                 nullptr, nullptr };
    if constexpr (Plane<R1, R2>::fits)
    {
        l.plane_r2c = launch_plane_r2c<R1, R2>;
        l.plane_c2r = launch_plane_c2r<R1, R2>;
    }
    return l;
}

} // namespace fftr

} // namespace nbx

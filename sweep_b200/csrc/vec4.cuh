// vec4.cuh -- four neighbouring x cells per thread: aligned 16-byte loads of
// pitched rows and the staggered differences on them.
//
// A thread of the kernels built on this owns the cells x .. x + 3 with x a
// multiple of 4 of a pitched row (pitch a multiple of 8 floats, so every row
// starts on a 32-byte sector).  A tap along y or z is one 16-byte load; the
// taps along x come from a window of the neighbouring groups.  Compared with
// one cell per thread this issues a quarter of the load instructions and of
// the index arithmetic, which is what bounded the one-cell kernels.
#pragma once

#include "common.cuh"

namespace sweep {
namespace v4 {

struct F4 {
    float v[4];
};

__device__ __forceinline__ F4 from(float4 t) { return F4{{t.x, t.y, t.z, t.w}}; }
// read-only in this kernel
__device__ __forceinline__ F4 ldg(const float* p) { return from(__ldg(reinterpret_cast<const float4*>(p))); }
// read and written in this kernel (by this thread only)
__device__ __forceinline__ F4 ld(const float* p) { return from(*reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ void st(float* p, const F4& a)
{
    *reinterpret_cast<float4*>(p) = make_float4(a.v[0], a.v[1], a.v[2], a.v[3]);
}
__device__ __forceinline__ F4 splat(float a) { return F4{{a, a, a, a}}; }

// Groups of 4 cells a window needs below / above the thread's own for taps
// reaching `n` cells out.
constexpr int groups(int n) { return (n + 3) / 4; }

// w[0 .. 4 (LO + 1 + HI)) = cells x - 4 LO .. x + 3 + 4 HI of the row at p
template <int LO, int HI>
__device__ __forceinline__ void window(const float* p, float (&w)[4 * (LO + 1 + HI)])
{
#pragma unroll
    for (int j = 0; j < LO + 1 + HI; ++j) {
        const F4 t = ldg(p + 4 * (j - LO));
#pragma unroll
        for (int l = 0; l < 4; ++l) w[4 * j + l] = t.v[l];
    }
}

// Staggered differences of half-width M with weights c[1..M]:
//   PLUS   sum_k c_k (u(k) - u(1 - k))      (to the half cell above)
//   else   sum_k c_k (u(k - 1) - u(-k))     (to the half cell below)
// row(k): the four cells k rows (or planes) away.
template <int M, bool PLUS, class R>
__device__ __forceinline__ F4 diff(const R& row, const float* c, float inv)
{
    F4 g;
#pragma unroll
    for (int k = 1; k <= M; ++k) {
        const F4 a = row(PLUS ? k : k - 1), b = row(PLUS ? 1 - k : -k);
#pragma unroll
        for (int l = 0; l < 4; ++l) g.v[l] = k == 1 ? c[1] * (a.v[l] - b.v[l]) : g.v[l] + c[k] * (a.v[l] - b.v[l]);
    }
#pragma unroll
    for (int l = 0; l < 4; ++l) g.v[l] *= inv;
    return g;
}

// the same along x, on a window whose element O is the thread's first cell
template <int M, bool PLUS, int O, int N>
__device__ __forceinline__ F4 diff_x(const float (&w)[N], const float* c, float inv)
{
    F4 g;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        float a = 0.f;
#pragma unroll
        for (int k = 1; k <= M; ++k) {
            const float d = PLUS ? w[O + l + k] - w[O + l + 1 - k] : w[O + l + k - 1] - w[O + l - k];
            a = k == 1 ? c[1] * d : a + c[k] * d;
        }
        g.v[l] = a * inv;
    }
    return g;
}

// window groups below / above for a PLUS or minus difference of half-width M
template <int M, bool PLUS>
struct Span {
    static constexpr int LO = groups(PLUS ? M - 1 : M), HI = groups(PLUS ? M : M - 1);
    static constexpr int N = 4 * (LO + 1 + HI), O = 4 * LO;
};

template <int M, bool PLUS>
__device__ __forceinline__ F4 diff_row(const float* p, const float* c, float inv)
{
    using S = Span<M, PLUS>;
    float w[S::N];
    window<S::LO, S::HI>(p, w);
    return diff_x<M, PLUS, S::O>(w, c, inv);
}

template <int M, bool PLUS>
__device__ __forceinline__ F4 diff_col(const float* p, int stride, const float* c, float inv)
{
    return diff<M, PLUS>([&](int k) { return ldg(p + k * stride); }, c, inv);
}

// staggered first-derivative weights of half-width M (the closed form
// a_m = (-1)^(m+1) / (2m - 1) prod_{n != m} |(2n-1)^2 / ((2n-1)^2 - (2m-1)^2)|,
// reference operators/staggered.cuh), each rounded from the exact ratio
inline void staggered_weights(int M, float* c)
{
    for (int m = 1; m <= M; ++m) {
        long long num = 1, den = 2 * m - 1;
        for (int n = 1; n <= M; ++n) {
            if (n == m) continue;
            const long long a = (long long)(2 * n - 1) * (2 * n - 1), q = (long long)(2 * m - 1) * (2 * m - 1);
            num *= a;
            den *= a > q ? a - q : q - a;
        }
        const double v = (double)num / (double)den;
        c[m] = (float)((m % 2 == 1) ? v : -v);
    }
}

}  // namespace v4
}  // namespace sweep

// fft_pair.cuh -- block-wide inverse FFT of PAIRS of transforms on
// packed FP32 arithmetic (fma/add/mul .f32x2 of sm_100a).
//
// Radix 16 with one last stage of radix 2, 4 or 8 where the size needs it;
// T = N/16 threads per pair, 16 points in registers.  Every register pair
// holds the same real or imaginary part of TWO transforms of one size, so
// each add, multiply and FMA of the butterflies serves both.
// The packed instructions run at the FP32 lanes' rate (measured: 128 lanes
// per clock and SM either way), so what they save is issue slots: half of
// the arithmetic ones, and half of the shared-memory ones too, since an
// element (re, im of both transforms) moves as one 16-byte access.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "fft_smem.cuh"

namespace msosm {
namespace pairfft {

// two floats, the same quantity of transform 0 (low half) and 1
typedef unsigned long long f2;

__device__ __forceinline__ f2 pk(float a, float b)
{
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 upk(f2 v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f2 dup(float a) { return pk(a, a); }
__device__ __forceinline__ f2 add2(f2 a, f2 b)
{
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b)
{
    f2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b)
{
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c)
{
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// complex values of both transforms
struct c2 {
    f2 re, im;
};
__device__ __forceinline__ c2 cadd(c2 a, c2 b) { return {add2(a.re, b.re), add2(a.im, b.im)}; }
__device__ __forceinline__ c2 csub(c2 a, c2 b) { return {sub2(a.re, b.re), sub2(a.im, b.im)}; }
// a + s b and a - s b, s real
__device__ __forceinline__ c2 caxpy(float s, c2 b, c2 a)
{
    const f2 k = dup(s);
    return {fma2(k, b.re, a.re), fma2(k, b.im, a.im)};
}
// a + SIGN i s b
template <int SIGN>
__device__ __forceinline__ c2 caxpy_i(float s, c2 b, c2 a)
{
    return {fma2(dup(SIGN > 0 ? -s : s), b.im, a.re), fma2(dup(SIGN > 0 ? s : -s), b.re, a.im)};
}
// a + SIGN i b
template <int SIGN>
__device__ __forceinline__ c2 cadd_i(c2 a, c2 b)
{
    if constexpr (SIGN > 0)
        return {sub2(a.re, b.im), add2(a.im, b.re)};
    else
        return {add2(a.re, b.im), sub2(a.im, b.re)};
}
// v * (w.x + i w.y), the same w for both transforms: eight scalar operations.
// Packed ones want w.x, w.y twice each; copied into register pairs that was
// 2.3 % slower at 4096 points, read twice from tables 3 %.
__device__ __forceinline__ c2 ctw(c2 v, float wx, float wy)
{
    const float2 r = upk(v.re), i = upk(v.im);
    return {pk(r.x * wx - i.x * wy, r.y * wx - i.y * wy), pk(r.x * wy + i.x * wx, r.y * wy + i.y * wx)};
}

__device__ __forceinline__ void dft4(c2 &x0, c2 &x1, c2 &x2, c2 &x3)
{
    const c2 a = cadd(x0, x2), b = csub(x0, x2), c = cadd(x1, x3), e = csub(x1, x3);
    x0 = cadd(a, c);
    x2 = csub(a, c);
    x1 = cadd_i<+1>(b, e);
    x3 = cadd_i<-1>(b, e);
}

// x[t] = X[4 t'] combinations of four values of which 1..3 still lack the
// factor k1 (1 and 3) or k2 (2): a0, k1 u1, k2 u2, k1 u3
__device__ __forceinline__ void dft4_scaled(c2 a0, c2 u1, c2 u2, c2 u3, float k1, float k2, c2 &x0, c2 &x1, c2 &x2,
                                            c2 &x3)
{
    const c2 p = caxpy(k2, u2, a0), q = caxpy(-k2, u2, a0), e = cadd(u1, u3), f = csub(u1, u3);
    x0 = caxpy(k1, e, p);
    x2 = caxpy(-k1, e, p);
    x1 = caxpy_i<+1>(k1, f, q);
    x3 = caxpy_i<-1>(k1, f, q);
}

__device__ __forceinline__ void dft2(c2 *v)
{
    const c2 a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
}

constexpr float kR2 = 0.70710678118654752440f;  // 1 / sqrt 2
constexpr float kC1 = 0.92387953251128675613f;  // cos(pi / 8)
constexpr float kT1 = 0.41421356237309504880f;  // tan(pi / 8)

// (1 + i) a
__device__ __forceinline__ c2 one_i(c2 a) { return cadd_i<+1>(a, a); }
// (-1 + i) a
__device__ __forceinline__ c2 mone_i(c2 a) { return {sub2(mul2(dup(-1.f), a.re), a.im), sub2(a.re, a.im)}; }
// (1 + i t) a and (t + i) a
__device__ __forceinline__ c2 one_it(float t, c2 a) { return caxpy_i<+1>(t, a, a); }
__device__ __forceinline__ c2 t_i(float t, c2 a)
{
    const f2 k = dup(t);
    return {sub2(mul2(k, a.re), a.im), fma2(k, a.im, a.re)};
}

__device__ __forceinline__ void dft4v(c2 *v) { dft4(v[0], v[1], v[2], v[3]); }

__device__ __forceinline__ void dft8(c2 *v)
{
    c2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    c2 o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
    dft4(e0, e1, e2, e3);
    dft4(o0, o1, o2, o3);
    // W8^1 = (1 + i)/sqrt2, W8^2 = i, W8^3 = (-1 + i)/sqrt2
    const c2 u1 = one_i(o1), u3 = mone_i(o3);
    v[0] = cadd(e0, o0);
    v[4] = csub(e0, o0);
    v[1] = caxpy(kR2, u1, e1);
    v[5] = caxpy(-kR2, u1, e1);
    v[2] = cadd_i<+1>(e2, o2);
    v[6] = cadd_i<-1>(e2, o2);
    v[3] = caxpy(kR2, u3, e3);
    v[7] = caxpy(-kR2, u3, e3);
}

// 16 points: four radix-4 butterflies, twiddles W16^(qs) with their common
// factor (cos pi/8 or 1/sqrt 2) left to the FMAs of the second radix-4 level:
// 142 packed operations instead of 160
__device__ __forceinline__ void dft16(c2 *v)
{
#pragma unroll
    for (int q = 0; q < 4; ++q)
        dft4(v[q], v[q + 4], v[q + 8], v[q + 12]);
    c2 o[16];
    o[0] = v[0];
    o[4] = v[1];
    o[8] = v[2];
    o[12] = v[3];
    dft4(o[0], o[4], o[8], o[12]);
    // s = 1: W^1 = C(1 + iT), W^2 = R(1 + i), W^3 = C(T + i)
    dft4_scaled(v[4], one_it(kT1, v[5]), one_i(v[6]), t_i(kT1, v[7]), kC1, kR2, o[1], o[5],
                      o[9], o[13]);
    // s = 2: W^2, W^4 = i, W^6 = R(-1 + i)
    {
        const c2 u1 = one_i(v[9]), u3 = mone_i(v[11]);
        const c2 p = cadd_i<+1>(v[8], v[10]), q = cadd_i<-1>(v[8], v[10]), e = cadd(u1, u3), f = csub(u1, u3);
        o[2] = caxpy(kR2, e, p);
        o[10] = caxpy(-kR2, e, p);
        o[6] = caxpy_i<+1>(kR2, f, q);
        o[14] = caxpy_i<-1>(kR2, f, q);
    }
    // s = 3: W^3 = C(T + i), W^6 = R(-1 + i), W^9 = -C(1 + iT)
    {
        const c2 u1 = t_i(kT1, v[13]), u2 = mone_i(v[14]), u3 = one_it(kT1, v[15]);
        const c2 p = caxpy(kR2, u2, v[12]), q = caxpy(-kR2, u2, v[12]), e = csub(u1, u3), f = cadd(u1, u3);
        o[3] = caxpy(kC1, e, p);
        o[11] = caxpy(-kC1, e, p);
        o[7] = caxpy_i<+1>(kC1, f, q);
        o[15] = caxpy_i<-1>(kC1, f, q);
    }
#pragma unroll
    for (int i = 0; i < 16; ++i)
        v[i] = o[i];
}

template <int R>
__device__ __forceinline__ void dft(c2 *v)
{
    if constexpr (R == 2)
        dft2(v);
    else if constexpr (R == 4)
        dft4v(v);
    else if constexpr (R == 8)
        dft8(v);
    else
        dft16(v);
}

__device__ __forceinline__ float4 to4(c2 v)
{
    const float2 r = upk(v.re), i = upk(v.im);
    return make_float4(r.x, r.y, i.x, i.y);
}
__device__ __forceinline__ c2 from4(float4 v) { return {pk(v.x, v.y), pk(v.z, v.w)}; }

// The transform is done in place (decimation in frequency): stage s
// transforms digit s of the element index, most significant first, and writes
// its result back to the same places, so a stage needs one barrier (before
// its loads) and a thread goes from its loads through its butterfly to its
// stores without one.  The radices are 16, 16, .. and RL last (FftShape); T
// threads hold 16 elements each.
//
//   n = d0 N/16 + rest,  rest = d1 N/256 + ..   input element
//   m = e0 + 16 e1 + ..                         output element (e: digits of the result)
//
// Stage 0: butterfly t = rest (element t + r N/16 in register r).  Stage s:
// butterfly j = e0 + 16 e1 + .. + 16^s rest, so that the last stage's outputs
// come in natural order, m = j + r N/R.  After stages 0 .. NST-3 the value
// with result digit e is multiplied by W_L^(e rest), L the sub-transform's
// length N/16^s; the factors due after stage NST-2 are applied to the last
// stage's inputs instead (R - 1 of R, as rest is then the digit itself).
//
// Element index i sits at i + i / (N/16), one pad per value of e0: the lanes of a
// quarter warp differ in e0 (consecutive i in stage 0), so its eight 16-byte
// accesses meet eight different bank groups.
template <int LOG2N>
struct PairFft {
    using F = FftShape<LOG2N>;
    static constexpr int N = F::N, T = F::T, NST = F::NST, LEAD = N / 16;
    // elements of one pair's buffer; 64 points: two pairs share a quarter warp
    static constexpr int SMEM = N + 16 + (N == 64 ? 4 : 0);
    __host__ __device__ static constexpr int len(int s) { return N >> (4 * s); }  // L of stage s < NS16
    __host__ __device__ static constexpr int stride(int s) { return s < F::NS16 ? N >> (4 * (s + 1)) : 1; }
    // words (floats) of a thread's twiddles before or after stage s: 15 complex
    // values after stages 0 .. NST-3; before the last stage (R - 1) for each
    // of its 16/R butterflies
    __host__ __device__ static constexpr int words(int s)
    {
        return s == NST - 1 ? 2 * (16 - 16 / F::radix(s)) : (s < NST - 2 ? 30 : 0);
    }
};

// place of butterfly j's element 0 at stage S >= 1
template <int LOG2N, int S>
__device__ __forceinline__ int inplace_base(int j)
{
    using P = PairFft<LOG2N>;
    int at = (j & 15) * (P::LEAD + 1);
    if constexpr (S >= 2)
        at += ((j >> 4) & 15) * (P::N >> 8);
    if constexpr (S >= 3)
        at += ((j >> 8) & 15) * (P::N >> 12);
    return at + (j >> (4 * S));  // rest
}

template <int LOG2N, int S>
__device__ __forceinline__ void stage_load(c2 (&v)[16], const float4 *__restrict__ buf, int tid)
{
    using P = PairFft<LOG2N>;
    constexpr int R = P::F::radix(S), B = 16 / R;
    static_assert(S >= 1, "stage 0 reads registers");
#pragma unroll
    for (int q = 0; q < B; ++q) {
        const float4 *p = buf + inplace_base<LOG2N, S>(tid + q * P::T);
#pragma unroll
        for (int r = 0; r < R; ++r)
            v[q * R + r] = from4(p[r * P::stride(S)]);
    }
}

template <int LOG2N, int S>
__device__ __forceinline__ void stage_store(const c2 (&v)[16], float4 *__restrict__ buf, int tid)
{
    using P = PairFft<LOG2N>;
    static_assert(S < P::NST - 1 && P::F::radix(S) == 16, "only radix-16 stages store");
    float4 *p = S == 0 ? buf + tid : buf + inplace_base<LOG2N, S>(tid);
#pragma unroll
    for (int r = 0; r < 16; ++r)
        p[r * (S == 0 ? P::LEAD + 1 : P::stride(S))] = to4(v[r]);
}

// This thread's twiddles of stage S (PairFft::words), from a table tw[e] =
// exp(2 pi i e / NTAB) (NTAB a multiple of N); further words are zero.
template <int LOG2N, int S, int NTAB>
__device__ __forceinline__ void stage_twiddles(float (&w)[32], int tid, const float2 *__restrict__ tw)
{
    using P = PairFft<LOG2N>;
    constexpr int R = P::F::radix(S), B = 16 / R;
    if constexpr (S == P::NST - 1) {
        // input r of butterfly j: W_L^(e r), L = 16 R, e the last digit done
#pragma unroll
        for (int q = 0; q < B; ++q) {
            const int e = ((tid + q * P::T) >> (4 * (S - 1))) & 15;
#pragma unroll
            for (int r = 1; r < R; ++r) {
                const float2 x = __ldg(&tw[e * r * (NTAB / (16 * R))]);
                w[2 * (q * (R - 1) + r - 1)] = x.x;
                w[2 * (q * (R - 1) + r - 1) + 1] = x.y;
            }
        }
    } else {
        const int rest = tid >> (4 * S);
#pragma unroll
        for (int e = 1; e < 16; ++e) {
            const float2 x = __ldg(&tw[e * rest * (NTAB / P::len(S))]);
            w[2 * e - 2] = x.x;
            w[2 * e - 1] = x.y;
        }
    }
#pragma unroll
    for (int i = P::words(S); i < 32; ++i)
        w[i] = 0.f;
}

// result digit e of a stage 0 .. NST-3: times its twiddle
__device__ __forceinline__ void twiddle_out(c2 (&v)[16], const float (&w)[32])
{
#pragma unroll
    for (int e = 1; e < 16; ++e)
        v[e] = ctw(v[e], w[2 * e - 2], w[2 * e - 1]);
}

// The last stage: input twiddles, butterflies.  Register slot q R + r then
// holds output m = tid + q T + r N/R (last_out_index).
template <int LOG2N>
__device__ __forceinline__ void last_stage(c2 (&v)[16], const float (&w)[32])
{
    using F = FftShape<LOG2N>;
    constexpr int R = F::radix(F::NST - 1), B = 16 / R;
#pragma unroll
    for (int q = 0; q < B; ++q) {
#pragma unroll
        for (int r = 1; r < R; ++r) {
            const int i = q * (R - 1) + r - 1;
            v[q * R + r] = ctw(v[q * R + r], w[2 * i], w[2 * i + 1]);
        }
        dft<R>(&v[q * R]);
    }
}

}  // namespace pairfft
}  // namespace msosm

// cnn.cu -- the DM-proposal network: a small 1-D CNN over coarse-DM folded
// profiles, trained and run with these kernels (msosm_cnn_* of msosm_b200.h).
//
// Input [B][Cin][L]: the folded profiles of Cin coarse DM trials, L phase
// bins.  `layers` circular ("same", wrapping in phase) convolutions of
// `channels` outputs and odd kernel K, each with ReLU; the mean over phase;
// two linear heads, a detection logit and a DM offset.  Weights are held in
// FP32 (the optimiser's copy) and used rounded to bf16; every product is
// accumulated in FP32.  Loss: the logistic loss of the logit, plus dm_weight
// times the mean over positive samples of the squared offset error.  Every
// reduction runs in a fixed order, so a step is deterministic.
//
// Parameter vector (one FP32 array): per layer the weights [C_out][C_in][K]
// and biases [C_out]; then the detection head's weights [C] and bias, then
// the offset head's weights [C] and bias.
#include "msosm_b200.h"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <new>
#include <random>
#include <string>
#include <type_traits>
#include <vector>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "fft_pair.cuh"
#include "kernels.hpp"

using namespace msosm;

namespace {

constexpr int kCoBlock = 8;  // output (or input) channels a thread accumulates

__device__ __forceinline__ void cp_async16(float *dst, const float *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async4(float *dst, const float *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

// Convolutions, forward and backward-data: one thread accumulates kCoBlock
// output channels x kT consecutive phases, in pairs of channels (packed FP32:
// two weights, one input value twice), so that per input channel and tap it
// reads two 16-byte weight vectors (the same for all threads of a channel
// group) for 32 packed FMAs; the inputs of all taps are four 16-byte reads.
// Bound by the FP32 lanes.  A block of 64 threads (16 across 128 phases x 4
// across 32 channels) makes 512 blocks for 256 samples; blocks of one warp for
// half the channels, 1024 of them, level the SMs better but read every input
// twice (33 us).  Input channels pass through two shared-memory buffers
// kCiChunk at a time, filled by cp.async from weights laid out as they are
// read (pack_weight).  256 samples x 256 phases, 7 taps, 32 -> 32 channels: 27
// us; 92 before (one shared-memory read per FMA, a block's whole input loaded
// first), 46 with four phases a thread and buffers filled between barriers.
constexpr int kT = 8;
constexpr int kCiChunk = 16;

// a block's input row in shared memory: phase tb + i at kXLead + i, so that
// its 16-byte vectors lie as in memory; the taps reach K/2 to either side
constexpr int kXLead = 8;
__host__ __device__ constexpr int conv_xw(int tt) { return kT * tt + 2 * kXLead + 4; }

// A block: tt threads across the phases, cg across the channels; 64 threads,
// or fewer for few channels or where the weights of that many channels do not
// fit (32 phases, 15 taps, 120 channels and more: half of the channel groups).
struct ConvShape {
    int tt, cg;
    ConvShape(int channels, int L, int K)
    {
        tt = L > 64 ? 16 : (L > 32 ? 8 : 4);
        cg = channels / kCoBlock < 64 / tt ? channels / kCoBlock : 64 / tt;
        while (cg > 1 && smem(K) > kConvSmemMax)
            cg = (cg + 1) / 2;
    }
    // both stages: kCiChunk input rows and their weights
    size_t smem(int K) const { return sizeof(float) * 2 * kCiChunk * ((size_t)conv_xw(tt) + (size_t)K * kCoBlock * cg); }
    static constexpr size_t kConvSmemMax = 227 * 1024;  // a block's share of sm_100a
};

using pairfft::f2;

// Forward: y[b][co][t] = relu(bias[co] + sum_ci sum_k w[co][ci][k] x[b][ci][t + k - p]),
// w as [ci][k][co].  BWD: dx[b][ci][s] = (act > 0) sum_co sum_k w[co][ci][k]
// g[b][co][s + p - k], w as [co][K - 1 - k][ci] (Cin: channels of g, Cout:
// channels of dx).  Phases wrap.  vec: `in` is 16-byte aligned.
template <int K, bool BWD>
__global__ void __launch_bounds__(64) conv_kernel(const float *__restrict__ in, int Cin, int L,
                                                  const float *__restrict__ w, const float *__restrict__ bias,
                                                  int Cout, ConvShape shape, int vec, const float *__restrict__ act,
                                                  float *__restrict__ out)
{
    extern __shared__ __align__(16) float smc[];
    constexpr int p = K / 2, LEAD = (p + 3) / 4 * 4;  // the thread's window starts LEAD before its phases
    static_assert(LEAD <= kXLead, "halo");
    constexpr int XN = (LEAD - p + K + kT - 1 + 3) / 4;
    const int tt = shape.tt, cg = shape.cg, xw = conv_xw(tt), wp = kCoBlock * cg;
    const int stage = kCiChunk * (xw + K * wp);  // floats: inputs [kCiChunk][xw], weights [kCiChunk K][wp]
    const int b = blockIdx.x, co0 = blockIdx.y * cg * kCoBlock, tb = blockIdx.z * tt * kT;
    const int ti = threadIdx.x % tt, gi = threadIdx.x / tt;
    const int co = co0 + gi * kCoBlock, t = tb + ti * kT;
    const int nco = min(wp, Cout - co0), n = min(kT * tt, L - tb);  // multiples of 8 and of 32
    const int chunks = (Cin + kCiChunk - 1) / kCiChunk;
    auto fetch = [&](int q) {
        if (q < chunks) {
            const int c0 = q * kCiChunk, cc = min(kCiChunk, Cin - c0);
            float *xs = smc + (q & 1) * stage, *ws = xs + kCiChunk * xw;
            const float *src = in + ((size_t)b * Cin + c0) * L;
            if (vec) {
                for (int e = threadIdx.x; e < cc * (n / 4); e += blockDim.x) {
                    const int c = e / (n / 4), j = 4 * (e - c * (n / 4));
                    cp_async16(xs + c * xw + kXLead + j, src + (size_t)c * L + tb + j);
                }
            } else {
                for (int e = threadIdx.x; e < cc * n; e += blockDim.x) {
                    const int c = e / n, j = e - c * n;
                    cp_async4(xs + c * xw + kXLead + j, src + (size_t)c * L + tb + j);
                }
            }
            for (int e = threadIdx.x; e < cc * (K - 1); e += blockDim.x) {
                const int c = e / (K > 1 ? K - 1 : 1), h = e - c * (K - 1);
                const int j = h < p ? h - p : n + h - p;  // p phases before, p after
                int ph = tb + j;
                ph += ph < 0 ? L : 0;
                ph -= ph >= L ? L : 0;
                cp_async4(xs + c * xw + kXLead + j, src + (size_t)c * L + ph);
            }
            const float *wq = w + (size_t)c0 * K * Cout + co0;
            for (int e = threadIdx.x; e < cc * K * (nco / 4); e += blockDim.x) {
                const int r = e / (nco / 4), j = 4 * (e - r * (nco / 4));
                cp_async16(ws + r * wp + j, wq + (size_t)r * Cout + j);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    f2 acc[kCoBlock / 2][kT];
#pragma unroll
    for (int j = 0; j < kCoBlock / 2; ++j) {
        const f2 z = BWD || co >= Cout ? pairfft::pk(0.f, 0.f) : pairfft::pk(bias[co + 2 * j], bias[co + 2 * j + 1]);
#pragma unroll
        for (int u = 0; u < kT; ++u)
            acc[j][u] = z;
    }
    fetch(0);
    for (int q = 0; q < chunks; ++q) {
        fetch(q + 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const int cc = min(kCiChunk, Cin - q * kCiChunk);
        const float *xs = smc + (q & 1) * stage;
        const float *xr = xs + kXLead - LEAD + ti * kT, *wr = xs + kCiChunk * xw + gi * kCoBlock;
        for (int c = 0; c < cc; ++c, xr += xw, wr += K * wp) {
            float x[4 * XN];
#pragma unroll
            for (int i = 0; i < XN; ++i) {
                const float4 v = reinterpret_cast<const float4 *>(xr)[i];
                x[4 * i] = v.x;
                x[4 * i + 1] = v.y;
                x[4 * i + 2] = v.z;
                x[4 * i + 3] = v.w;
            }
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const ulonglong2 w01 = *reinterpret_cast<const ulonglong2 *>(wr + k * wp);
                const ulonglong2 w23 = *reinterpret_cast<const ulonglong2 *>(wr + k * wp + 4);
                const f2 wv[4] = {w01.x, w01.y, w23.x, w23.y};
#pragma unroll
                for (int u = 0; u < kT; ++u) {
                    const f2 xv = pairfft::dup(x[LEAD - p + k + u]);
#pragma unroll
                    for (int j = 0; j < kCoBlock / 2; ++j)
                        acc[j][u] = pairfft::fma2(wv[j], xv, acc[j][u]);
                }
            }
        }
        __syncthreads();  // before the buffer is filled again
    }
    if (co >= Cout || t >= L)
        return;
#pragma unroll
    for (int j = 0; j < kCoBlock; ++j) {
        const size_t at = ((size_t)b * Cout + co + j) * L + t;
        float v[kT];
#pragma unroll
        for (int u = 0; u < kT; ++u) {
            const float2 a = pairfft::upk(acc[j / 2][u]);
            v[u] = j & 1 ? a.y : a.x;
        }
#pragma unroll
        for (int u = 0; u < kT; u += 4) {
            float4 o;
            if constexpr (BWD) {
                const float4 m = *reinterpret_cast<const float4 *>(act + at + u);
                o = make_float4(m.x > 0.f ? v[u] : 0.f, m.y > 0.f ? v[u + 1] : 0.f, m.z > 0.f ? v[u + 2] : 0.f,
                                m.w > 0.f ? v[u + 3] : 0.f);
            } else {
                o = make_float4(fmaxf(v[u], 0.f), fmaxf(v[u + 1], 0.f), fmaxf(v[u + 2], 0.f), fmaxf(v[u + 3], 0.f));
            }
            *reinterpret_cast<float4 *>(out + at + u) = o;
        }
    }
}

// Weight gradients: dw[co][ci][k] = sum_b sum_t g[b][co][t] a[b][ci][t + k - p]
// and db[co] = sum_b sum_t g[b][co][t].  A block sums a group of samples for 32
// output x 8 input channels: each lane holds 4 output x 2 input channels x K
// taps in registers (co = lane % 8 + 8 i, ci = 2 (lane / 8) + {0, 1}, the two
// input channels as a packed pair), the four warps a quarter of the phases
// each, so that 9 16-byte reads of shared memory feed 16 K packed FMAs.  Warps are added in order, groups by wgrad_reduce_kernel in
// order.
// Bound by the FP32 lanes and shared memory.  256 samples x 256 phases, 64 ->
// 32 channels, 7 taps: 60 us, 820 before (one block per (co, ci), every
// product's operands read from memory).
// The phases pass in chunks of kWgT through kWgStages buffers filled by
// cp.async (one buffer filled between barriers took 79 us instead).
constexpr int kWgCo = 32, kWgCi = 8, kWgT = 64, kWgStages = 3;
constexpr int kWgGs = kWgT + 4;   // row strides: the eight (four) rows of a read in different banks
constexpr int kWgAs = 2 * (kWgT + 18);  // two channels interleaved
constexpr int kWgStage = kWgCo * kWgGs + kWgCi / 2 * kWgAs;  // floats

template <int K>
__global__ void __launch_bounds__(128, K <= 7 ? 4 : 2) conv_wgrad_kernel(const float *__restrict__ g, int Co,
                                                         const float *__restrict__ a, int Ci, int B, int L, int groups,
                                                         float *__restrict__ part)
{
    static_assert(2 * (kWgT + K + 2) <= kWgAs, "a phase chunk with its halo");
    extern __shared__ __align__(16) float smc[];
    constexpr int p = K / 2;
    const int ci0 = blockIdx.x * kWgCi, co0 = blockIdx.y * kWgCo, grp = blockIdx.z;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lg = lane & 7, la = lane >> 3;
    // units of one sample x one phase chunk; this group's
    const int nt = (L + kWgT - 1) / kWgT;
    const int u0 = (int)((long long)B * nt * grp / groups), u1 = (int)((long long)B * nt * (grp + 1) / groups);
    const bool with_bias = blockIdx.x == 0;
    f2 acc2[4][K];
    float ab[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        ab[i] = 0.f;
#pragma unroll
        for (int k = 0; k < K; ++k)
            acc2[i][k] = pairfft::pk(0.f, 0.f);
    }
    auto fetch = [&](int u) {
        if (u < u1) {
            const int b = u / nt, tb = (u - b * nt) * kWgT, n = min(kWgT, L - tb);  // n a multiple of 32
            float *gs = smc + (u % kWgStages) * kWgStage, *as = gs + kWgCo * kWgGs;
#pragma unroll
            for (int i = 0; i < kWgCo * kWgT / 4 / 128; ++i) {
                const int v = threadIdx.x + 128 * i, r = v / (kWgT / 4), j = 4 * (v % (kWgT / 4));
                if (j < n) {
                    if (co0 + r < Co)
                        cp_async16(gs + r * kWgGs + j, g + ((size_t)b * Co + co0 + r) * L + tb + j);
                    else
                        *reinterpret_cast<float4 *>(gs + r * kWgGs + j) = make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
#pragma unroll
            for (int i = 0; i < kWgCi / 4; ++i) {
                const int r = warp + 4 * i;
                const float *src = a + ((size_t)b * Ci + ci0 + r) * L;
                for (int j = lane; j < n + K - 1; j += 32) {
                    int s = tb + j - p;
                    s += s < 0 ? L : 0;
                    s -= s >= L ? L : 0;
                    cp_async4(as + (r >> 1) * kWgAs + 2 * j + (r & 1), src + s);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int i = 0; i < kWgStages - 1; ++i)
        fetch(u0 + i);
    for (int u = u0; u < u1; ++u) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kWgStages - 2) : "memory");
        __syncthreads();  // unit u is in; everyone is done with the buffer fetched into next
        fetch(u + kWgStages - 1);
        const float *gs = smc + (u % kWgStages) * kWgStage, *as = gs + kWgCo * kWgGs;
        const int n = min(kWgT, L - (u % nt) * kWgT);
        for (int t = warp * (n / 4); t < (warp + 1) * (n / 4); t += 4) {
            float gv[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 v = *reinterpret_cast<const float4 *>(gs + (lg + 8 * i) * kWgGs + t);
                gv[i][0] = v.x;
                gv[i][1] = v.y;
                gv[i][2] = v.z;
                gv[i][3] = v.w;
            }
            // phases t .. t + K + 2 of both input channels
            f2 x[(K + 4) / 2 * 2];
#pragma unroll
            for (int i = 0; i < (K + 4) / 2; ++i) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(as + la * kWgAs + 2 * t + 4 * i);
                x[2 * i] = v.x;
                x[2 * i + 1] = v.y;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    const f2 gg = pairfft::dup(gv[i][v]);
#pragma unroll
                    for (int k = 0; k < K; ++k)
                        acc2[i][k] = pairfft::fma2(gg, x[k + v], acc2[i][k]);
                }
            if (with_bias)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    ab[i] += (gv[i][0] + gv[i][1]) + (gv[i][2] + gv[i][3]);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    float acc[4][2][K];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const float2 v = pairfft::upk(acc2[i][k]);
            acc[i][0][k] = v.x;
            acc[i][1][k] = v.y;
        }
    // warps 1 .. 3 onto warp 0, one after another
    for (int w = 1; w < 4; ++w) {
        __syncthreads();
        if (warp == w) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                smc[(8 * K + i) * 32 + lane] = ab[i];
#pragma unroll
                for (int q = 0; q < 2; ++q)
#pragma unroll
                    for (int k = 0; k < K; ++k)
                        smc[((i * 2 + q) * K + k) * 32 + lane] = acc[i][q][k];
            }
        }
        __syncthreads();
        if (warp == 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                ab[i] += smc[(8 * K + i) * 32 + lane];
#pragma unroll
                for (int q = 0; q < 2; ++q)
#pragma unroll
                    for (int k = 0; k < K; ++k)
                        acc[i][q][k] += smc[((i * 2 + q) * K + k) * 32 + lane];
            }
        }
    }
    if (warp != 0)
        return;
    // this group's row of partial sums: the weights, then the biases
    float *row = part + (size_t)grp * ((size_t)Co * Ci * K + Co);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int co = co0 + lg + 8 * i;
        if (co >= Co)
            continue;
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int k = 0; k < K; ++k)
                row[((size_t)co * Ci + ci0 + 2 * la + q) * K + k] = acc[i][q][k];
        if (with_bias && la == 0)
            row[(size_t)Co * Ci * K + co] = ab[i];
    }
}

// Partial rows of the layers' weight gradients: row r of layer l at part +
// offset[l] + r n, n = values[l] weights then biases, as they lie in the
// gradient at out[l].
constexpr int kMaxLayers = 16;

struct WgradRows {
    const float *part;
    float *grad;
    long long offset[kMaxLayers], out[kMaxLayers], values[kMaxLayers];
    int groups[kMaxLayers];
};

// Sum of the groups' rows of every layer (blockIdx.y) in one launch after the
// backward pass.  Eight slices of the rows per value, added in order, in FP64:
// in FP32 these few additions of nearly whole sums were most of a weight
// gradient's rounding (1.3e-7 of its size, 0.9e-7 now, last layer of the
// defaults).  Bound by
// latency: a launch per layer, each between two convolutions, took 5 - 7 us (a
// gradient of 256 samples and four layers 459 us, with one launch 442).
__global__ void __launch_bounds__(256) wgrad_reduce_kernel(const __grid_constant__ WgradRows rows)
{
    __shared__ double sums[8][32];
    const int lane = threadIdx.x & 31, sl = threadIdx.x >> 5, l = blockIdx.y, groups = rows.groups[l];
    const long long i = (long long)blockIdx.x * 32 + lane, n = rows.values[l];
    if ((long long)blockIdx.x * 32 >= n)
        return;
    const float *__restrict__ part = rows.part + rows.offset[l];
    double s = 0.0;
    if (i < n) {
#pragma unroll 4
        for (int g = sl; g < groups; g += 8)
            s += (double)part[(size_t)g * n + i];
    }
    sums[sl][lane] = s;
    __syncthreads();
    if (sl == 0 && i < n) {
#pragma unroll
        for (int k = 1; k < 8; ++k)
            s += sums[k][lane];
        rows.grad[rows.out[l] + i] = (float)s;
    }
}

// groups of the weight gradient's units: about four blocks per SM in all
inline int wgrad_groups(int Co, int Ci, int B)
{
    const int tiles = (Ci / kWgCi) * ((Co + kWgCo - 1) / kWgCo);
    const int n = 592 / tiles;
    return n < 1 ? 1 : (n > B ? B : n);
}

// go(std::integral_constant<int, K>) for the odd kernel widths
template <class G>
cudaError_t with_taps(int K, G &&go)
{
    switch (K) {
    case 1: return go(std::integral_constant<int, 1>{});
    case 3: return go(std::integral_constant<int, 3>{});
    case 5: return go(std::integral_constant<int, 5>{});
    case 7: return go(std::integral_constant<int, 7>{});
    case 9: return go(std::integral_constant<int, 9>{});
    case 11: return go(std::integral_constant<int, 11>{});
    case 13: return go(std::integral_constant<int, 13>{});
    case 15: return go(std::integral_constant<int, 15>{});
    default: return cudaErrorInvalidValue;
    }
}

template <bool BWD>
cudaError_t launch_conv(int K, const float *in, int Cin, int L, const float *w, const float *bias, int Cout, int B,
                        const float *act, float *out, cudaStream_t st)
{
    return with_taps(K, [&](auto taps) -> cudaError_t {
        constexpr int KK = decltype(taps)::value;
        const ConvShape shape(Cout, L, KK);
        const int cg = shape.cg, tt = shape.tt;
        const size_t sm = shape.smem(KK);
        auto k = conv_kernel<KK, BWD>;
        cudaError_t e = allow_smem(k, sm);
        if (e != cudaSuccess)
            return e;
        const dim3 grid(B, (Cout / kCoBlock + cg - 1) / cg, (L + kT * tt - 1) / (kT * tt));
        const int vec = (reinterpret_cast<uintptr_t>(in) & 15) == 0;
        k<<<grid, tt * cg, sm, st>>>(in, Cin, L, w, bias, Cout, shape, vec, act, out);
        return cudaGetLastError();
    });
}

// dw (then db) of one layer into its partial rows
cudaError_t launch_wgrad(int K, const float *g, int Co, const float *a, int Ci, int B, int L, float *part,
                         cudaStream_t st)
{
    return with_taps(K, [&](auto taps) -> cudaError_t {
        constexpr int KK = decltype(taps)::value;
        const int groups = wgrad_groups(Co, Ci, B);
        const size_t sm = sizeof(float) * kWgStages * kWgStage;
        auto k = conv_wgrad_kernel<KK>;
        cudaError_t e = allow_smem(k, sm);
        if (e != cudaSuccess)
            return e;
        k<<<dim3(Ci / kWgCi, (Co + kWgCo - 1) / kWgCo, groups), 128, sm, st>>>(g, Co, a, Ci, B, L, groups, part);
        return cudaGetLastError();
    });
}

// h[b][c] = mean over t of a[b][c][t] (warp w of the block takes channels w,
// w + warps, ...), then both heads' values of the sample from it (warp 0).
__global__ void __launch_bounds__(1024) pool_heads_kernel(const float *__restrict__ a, int C, int L,
                                                          const __nv_bfloat16 *__restrict__ wd,
                                                          const float *__restrict__ bd,
                                                          const __nv_bfloat16 *__restrict__ wr,
                                                          const float *__restrict__ br, float *__restrict__ h,
                                                          float *__restrict__ logit, float *__restrict__ offset)
{
    __shared__ float hs[256];
    const int b = blockIdx.x, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    for (int c = threadIdx.x >> 5; c < C; c += warps) {
        const float *r = a + ((size_t)b * C + c) * L;
        float s = 0.f;
#pragma unroll 4
        for (int t = lane; t < L; t += 32)
            s += r[t];
        for (int o = 16; o > 0; o >>= 1)
            s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0)
            h[b * C + c] = hs[c] = s / (float)L;
    }
    __syncthreads();
    if (threadIdx.x >= 32)
        return;
    // (FP64: a few hundred operations of one warp; the terms cancel, and what
    // their rounding leaves goes into the loss and every gradient)
    double lg = 0.0, of = 0.0;
    for (int c = lane; c < C; c += 32) {
        lg = fma((double)hs[c], (double)__bfloat162float(wd[c]), lg);
        of = fma((double)hs[c], (double)__bfloat162float(wr[c]), of);
    }
    for (int o = 16; o > 0; o >>= 1) {
        lg += __shfl_xor_sync(0xffffffffu, lg, o);
        of += __shfl_xor_sync(0xffffffffu, of, o);
    }
    if (lane == 0) {
        logit[b] = (float)(lg + (double)*bd);
        offset[b] = (float)(of + (double)*br);
    }
}

constexpr int kHeadThreads = 1024;  // at least max_batch

struct HeadArgs {
    const float *h;              // [B][C]
    const float *logit, *offset; // [B]
    const float *label, *target; // [B]
    float *dl, *dof;             // [B]: gradients of the logit and the offset
    float *gwd, *gbd, *gwr, *gbr;
    float *loss;                 // [1]
    int B, C;
    float dm_weight;
};

// The loss, its gradients by the heads' outputs and the heads' own gradients:
// one block, a thread to a sample (B <= blockDim.x); sums in a fixed order.
__global__ void __launch_bounds__(1024) heads_grad_kernel(HeadArgs a)
{
    extern __shared__ float hs[];  // [5][blockDim.x]: dlogit, doff, loss terms, two partial sums
    float *dl = hs, *dof = hs + blockDim.x, *lt = hs + 2 * blockDim.x;
    const int b = threadIdx.x;
    float lg = 0.f, y = 0.f, err = 0.f;
    bool pos = false;
    if (b < a.B) {
        lg = a.logit[b];
        y = a.label[b];
        pos = y > 0.5f;
        err = a.offset[b] - a.target[b];
    }
    // number of positive samples
    const float npos = fmaxf((float)__syncthreads_count(b < a.B && pos), 1.f);
    if (b < a.B) {
        const float sg = 1.f / (1.f + expf(-lg));
        a.dl[b] = dl[b] = (sg - y) / (float)a.B;
        a.dof[b] = dof[b] = pos ? a.dm_weight * 2.f * err / npos : 0.f;
        const float lo = fmaxf(lg, 0.f) - lg * y + log1pf(expf(-fabsf(lg)));
        lt[b] = lo / (float)a.B + (pos ? a.dm_weight * err * err / npos : 0.f);
    }
    __syncthreads();
    // weight gradients: as many slices of the samples as the block has room
    // for, slice s samples s, s + S, ..; the slices' sums added in order
    const int S = (int)blockDim.x / a.C;
    float *pd = lt + blockDim.x, *pr = pd + blockDim.x;
    const int sl = b / a.C, c = b - sl * a.C;
    if (sl < S) {
        float gd = 0.f, gr = 0.f;
#pragma unroll 8
        for (int i = sl; i < a.B; i += S) {
            const float hv = a.h[i * a.C + c];
            gd = fmaf(dl[i], hv, gd);
            gr = fmaf(dof[i], hv, gr);
        }
        pd[b] = gd;
        pr[b] = gr;
    }
    __syncthreads();
    if (b < a.C) {
        float gd = 0.f, gr = 0.f;
        for (int s = 0; s < S; ++s) {
            gd += pd[s * a.C + b];
            gr += pr[s * a.C + b];
        }
        a.gwd[b] = gd;
        a.gwr[b] = gr;
    }
    // the biases' gradients and the loss: one warp, lane-strided sums and a
    // butterfly
    if (b < 32) {
        float sd = 0.f, sr = 0.f, l = 0.f;
        for (int i = b; i < a.B; i += 32) {
            sd += dl[i];
            sr += dof[i];
            l += lt[i];
        }
        for (int o = 16; o > 0; o >>= 1) {
            sd += __shfl_xor_sync(0xffffffffu, sd, o);
            sr += __shfl_xor_sync(0xffffffffu, sr, o);
            l += __shfl_xor_sync(0xffffffffu, l, o);
        }
        if (b == 0) {
            *a.gbd = sd;
            *a.gbr = sr;
            *a.loss = l;
        }
    }
}

// g[b][c][t] = (a[b][c][t] > 0) dh[b][c] / L, dh[b][c] = dl[b] wd[c] + dof[b] wr[c]
// (the backward of the heads, the mean and ReLU), four phases a thread, n4 of
// them
__global__ void pool_bwd_kernel(const float *__restrict__ dl, const float *__restrict__ dof,
                                const __nv_bfloat16 *__restrict__ wd, const __nv_bfloat16 *__restrict__ wr,
                                const float4 *__restrict__ a, unsigned C, unsigned L4, unsigned n4, float len,
                                float4 *__restrict__ g)
{
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n4)
        return;
    const unsigned bc = i / L4, b = bc / C, c = bc - b * C;
    const float d = (dl[b] * __bfloat162float(wd[c]) + dof[b] * __bfloat162float(wr[c])) / len;
    const float4 v = a[i];
    g[i] = make_float4(v.x > 0.f ? d : 0.f, v.y > 0.f ? d : 0.f, v.z > 0.f ? d : 0.f, v.w > 0.f ? d : 0.f);
}

// The convolutions' weights as their kernels read them (float values of the
// bf16 rounding): per layer [ci][k][co] for the forward pass and, at the same
// offsets, [co][K - 1 - k][ci] for the backward one.
struct PackArgs {
    float *fwd, *bwd;
    int layers, C, Cin0, K;
};
__device__ __forceinline__ void pack_weight(const PackArgs &p, long long i, float v)
{
    const long long first = (long long)p.C * p.Cin0 * p.K + p.C, rest = (long long)p.C * p.C * p.K + p.C;
    const int l = i < first ? 0 : (int)((i - first) / rest) + 1;
    if (l >= p.layers)
        return;  // the heads
    const int ci_n = l == 0 ? p.Cin0 : p.C;
    const long long off = l == 0 ? 0 : first + (l - 1) * rest;
    const int e = (int)(i - off);
    if (e >= p.C * ci_n * p.K)
        return;  // a bias
    const int k = e % p.K, ci = e / p.K % ci_n, co = e / p.K / ci_n;
    p.fwd[off + ((long long)ci * p.K + k) * p.C + co] = v;
    p.bwd[off + ((long long)co * p.K + p.K - 1 - k) * ci_n + ci] = v;
}

// Adam on the FP32 parameters, then their bf16 copies
__global__ void adam_kernel(float *__restrict__ th, const float *__restrict__ g, float *__restrict__ m,
                            float *__restrict__ v, __nv_bfloat16 *__restrict__ q, long long n, float lr, float b1,
                            float b2, float c1, float c2, float eps, PackArgs pack)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float t = th[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    th[i] = t;
    q[i] = __float2bfloat16_rn(t);
    pack_weight(pack, i, __bfloat162float(q[i]));
}

__global__ void quantise_kernel(const float *__restrict__ th, __nv_bfloat16 *__restrict__ q, long long n,
                                PackArgs pack)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const __nv_bfloat16 v = __float2bfloat16_rn(th[i]);
        q[i] = v;
        pack_weight(pack, i, __bfloat162float(v));
    }
}

inline unsigned nblocks(long long n, int t) { return (unsigned)((n + t - 1) / t); }

msosm_status cfail(msosm_status s, const std::string &m)
{
    set_error_message(m.c_str());
    return s;
}

msosm_status ccuda(cudaError_t e, const char *what)
{
    cudaGetLastError();
    return cfail(e == cudaErrorMemoryAllocation ? MSOSM_ERR_OOM : MSOSM_ERR_CUDA,
                 std::string(what) + ": " + cudaGetErrorString(e));
}

bool on_device(const void *p)
{
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged;
}

}  // namespace

struct msosm_cnn {
    msosm_cnn_config cfg{};
    long long n = 0;                 // parameters
    std::vector<long long> w_off, b_off;  // per layer; then the heads at hd..
    long long wd_off = 0, bd_off = 0, wr_off = 0, br_off = 0;
    float *slab = nullptr;           // what all the buffers below lie in
    float *th = nullptr, *grad = nullptr, *m = nullptr, *v = nullptr;
    __nv_bfloat16 *q = nullptr;
    std::vector<float *> act;        // act[1..layers]: [max_batch][C][L]
    float *xin = nullptr, *lab = nullptr, *tgt = nullptr;  // staged host inputs
    float *part = nullptr;           // partial rows of the weight gradients, layer l's from part_off[l]
    std::vector<long long> part_off;
    float *g0 = nullptr, *g1 = nullptr;  // gradient ping-pong [max_batch][max(Cin, C)][L]
    float *wf = nullptr, *wb = nullptr;  // packed weights (PackArgs)
    float *h = nullptr, *dl = nullptr, *dof = nullptr, *logit = nullptr, *off = nullptr, *loss = nullptr;
    cudaStream_t st = nullptr;
    long long steps = 0;

    void release()
    {
        if (slab)
            cudaFree(slab);
        if (st)
            cudaStreamDestroy(st);
    }
};

namespace {

cudaError_t conv_forward(msosm_cnn *c, const float *x, int B)
{
    const msosm_cnn_config &g = c->cfg;
    const float *in = x;
    int ci = g.in_channels;
    for (int l = 0; l < g.layers; ++l) {
        cudaError_t e = launch_conv<false>(g.kernel, in, ci, g.length, c->wf + c->w_off[l], c->th + c->b_off[l],
                                           g.channels, B, nullptr, c->act[l + 1], c->st);
        if (e != cudaSuccess)
            return e;
        in = c->act[l + 1];
        ci = g.channels;
    }
    pool_heads_kernel<<<B, 32 * (g.channels < 32 ? g.channels : 32), 0, c->st>>>(
        c->act[g.layers], g.channels, g.length, c->q + c->wd_off, c->th + c->bd_off, c->q + c->wr_off,
        c->th + c->br_off, c->h, c->logit, c->off);
    return cudaGetLastError();
}

PackArgs pack_args(const msosm_cnn *c)
{
    return {c->wf, c->wb, c->cfg.layers, c->cfg.channels, c->cfg.in_channels, c->cfg.kernel};
}

// device copy of a [n] float input (host or device pointer)
const float *stage(msosm_cnn *c, const float *src, float *buf, size_t n, cudaError_t &e)
{
    if (on_device(src))
        return src;
    e = cudaMemcpyAsync(buf, src, sizeof(float) * n, cudaMemcpyHostToDevice, c->st);
    return buf;
}

msosm_status check_batch(const msosm_cnn *c, int B)
{
    if (!c)
        return cfail(MSOSM_ERR_BAD_ARG, "null network");
    if (B < 1 || B > c->cfg.max_batch)
        return cfail(MSOSM_ERR_BAD_ARG, "batch must be 1 .. max_batch");
    return MSOSM_OK;
}

}  // namespace

extern "C" {

msosm_status msosm_cnn_create(const msosm_cnn_config *cfg, unsigned long long seed, msosm_cnn **out)
{
    if (!cfg || !out)
        return cfail(MSOSM_ERR_BAD_ARG, "null argument");
    *out = nullptr;
    const msosm_cnn_config &g = *cfg;
    if (g.in_channels < 1 || g.in_channels > 256 || g.length < 32 || g.length > 1024 || g.length % 32 != 0 ||
        g.channels < kCoBlock || g.channels > 256 || g.channels % kCoBlock != 0 || g.in_channels % kCoBlock != 0 ||
        g.kernel < 1 || g.kernel > 15 || g.kernel % 2 == 0 || g.kernel > g.length || g.layers < 1 ||
        g.layers > kMaxLayers || g.max_batch < 1 || g.max_batch > 1024 || !(g.dm_weight >= 0.f))
        return cfail(MSOSM_ERR_BAD_ARG,
                     "cnn: in_channels and channels multiples of 8 (<= 256), length a multiple of 32 in 32 .. 1024, "
                     "odd kernel <= 15, 1 .. 16 layers, max_batch 1 .. 1024, dm_weight >= 0");
    // the accepted sizes are those whose widest layer, whole, fits 200 KB
    const int cmax = g.in_channels > g.channels ? g.in_channels : g.channels;
    const size_t sm = sizeof(float) * ((size_t)cmax * (g.length + g.kernel - 1) + (size_t)kCoBlock * cmax * g.kernel);
    if (sm > 200 * 1024)
        return cfail(MSOSM_ERR_UNSUPPORTED, "cnn: channels x length too large for one block's shared memory");
    if (msosm_device_count() == 0)
        return cfail(MSOSM_ERR_NO_DEVICE, "no CUDA device");
    msosm_cnn *c = new (std::nothrow) msosm_cnn;
    if (!c)
        return cfail(MSOSM_ERR_OOM, "host allocation");
    c->cfg = g;
    long long o = 0;
    int ci = g.in_channels;
    for (int l = 0; l < g.layers; ++l) {
        c->w_off.push_back(o);
        o += (long long)g.channels * ci * g.kernel;
        c->b_off.push_back(o);
        o += g.channels;
        ci = g.channels;
    }
    c->wd_off = o;
    o += g.channels;
    c->bd_off = o;
    o += 1;
    c->wr_off = o;
    o += g.channels;
    c->br_off = o;
    o += 1;
    c->n = o;
    // He-uniform initial weights (fan-in), zero biases, from a seeded engine
    std::vector<float> init((size_t)o, 0.f);
    std::mt19937_64 rng(seed);
    ci = g.in_channels;
    for (int l = 0; l < g.layers; ++l) {
        const double lim = std::sqrt(6.0 / (double)(ci * g.kernel));
        std::uniform_real_distribution<double> u(-lim, lim);
        for (long long i = 0; i < (long long)g.channels * ci * g.kernel; ++i)
            init[(size_t)(c->w_off[l] + i)] = (float)u(rng);
        ci = g.channels;
    }
    {
        const double lim = std::sqrt(3.0 / (double)g.channels);
        std::uniform_real_distribution<double> u(-lim, lim);
        for (int i = 0; i < g.channels; ++i) {
            init[(size_t)(c->wd_off + i)] = (float)u(rng);
            init[(size_t)(c->wr_off + i)] = (float)u(rng);
        }
    }
    const size_t B = (size_t)g.max_batch, L = (size_t)g.length;
    const size_t gmax = B * (size_t)cmax * L;
    cudaError_t e = cudaStreamCreateWithFlags(&c->st, cudaStreamNonBlocking);
    // one allocation for all float buffers, each 256-byte aligned
    std::vector<std::pair<float **, size_t>> slots;
    size_t total = 0;
    auto al = [&](float **p, size_t count) {
        slots.push_back({p, total});
        total += (count + 4 + 63) / 64 * 64;
    };
    al(&c->th, (size_t)o);
    al(&c->grad, (size_t)o);
    al(&c->m, (size_t)o);
    al(&c->v, (size_t)o);
    float *q = nullptr;
    al(&q, ((size_t)o + 1) / 2);
    c->act.assign(g.layers + 1, nullptr);
    for (int l = 1; l <= g.layers; ++l)
        al(&c->act[l], B * g.channels * L);
    al(&c->xin, B * (size_t)g.in_channels * L);
    al(&c->lab, B);
    al(&c->tgt, B);
    al(&c->g0, gmax);
    al(&c->g1, gmax);
    al(&c->h, B * g.channels);
    al(&c->dl, B);
    al(&c->dof, B);
    al(&c->wf, (size_t)o);
    al(&c->wb, (size_t)o);
    al(&c->logit, B);
    al(&c->off, B);
    al(&c->loss, 1);
    // partial rows of the weight gradients
    size_t prows = 0;
    for (int l = 0; l < g.layers; ++l) {
        const int cin = l == 0 ? g.in_channels : g.channels;
        const size_t n = (size_t)g.channels * cin * g.kernel + g.channels;
        c->part_off.push_back((long long)prows);
        prows += n * (size_t)wgrad_groups(g.channels, cin, g.max_batch);
    }
    al(&c->part, prows);
    if (e == cudaSuccess)
        e = cudaMalloc((void **)&c->slab, sizeof(float) * total);
    if (e == cudaSuccess) {
        for (const auto &sl : slots)
            *sl.first = c->slab + sl.second;
        c->q = reinterpret_cast<__nv_bfloat16 *>(q);
    }
    if (e != cudaSuccess) {
        msosm_status s = ccuda(e, "msosm_cnn_create");
        c->release();
        delete c;
        return s;
    }
    *out = c;
    msosm_status s = msosm_cnn_set_params(c, init.data());
    if (s != MSOSM_OK) {
        c->release();
        delete c;
        *out = nullptr;
    }
    return s;
}

msosm_status msosm_cnn_destroy(msosm_cnn *c)
{
    if (c) {
        if (c->st)
            cudaStreamSynchronize(c->st);
        c->release();
        delete c;
    }
    return MSOSM_OK;
}

msosm_status msosm_cnn_param_count(const msosm_cnn *c, size_t *count)
{
    if (!c || !count)
        return cfail(MSOSM_ERR_BAD_ARG, "null argument");
    *count = (size_t)c->n;
    return MSOSM_OK;
}

msosm_status msosm_cnn_get_params(msosm_cnn *c, float *params)
{
    if (!c || !params)
        return cfail(MSOSM_ERR_BAD_ARG, "null argument");
    cudaError_t e = cudaMemcpyAsync(params, c->th, sizeof(float) * c->n, cudaMemcpyDeviceToHost, c->st);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(c->st);
    return e == cudaSuccess ? MSOSM_OK : ccuda(e, "msosm_cnn_get_params");
}

msosm_status msosm_cnn_set_params(msosm_cnn *c, const float *params)
{
    if (!c || !params)
        return cfail(MSOSM_ERR_BAD_ARG, "null argument");
    cudaError_t e = cudaMemcpyAsync(c->th, params, sizeof(float) * c->n, cudaMemcpyDefault, c->st);
    if (e == cudaSuccess)
        e = cudaMemsetAsync(c->m, 0, sizeof(float) * c->n, c->st);
    if (e == cudaSuccess)
        e = cudaMemsetAsync(c->v, 0, sizeof(float) * c->n, c->st);
    if (e == cudaSuccess) {
        quantise_kernel<<<nblocks(c->n, 256), 256, 0, c->st>>>(c->th, c->q, c->n, pack_args(c));
        e = cudaGetLastError();
    }
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(c->st);
    c->steps = 0;
    return e == cudaSuccess ? MSOSM_OK : ccuda(e, "msosm_cnn_set_params");
}

msosm_status msosm_cnn_forward(msosm_cnn *c, const float *x, int batch, float *logit, float *offset)
{
    msosm_status s = check_batch(c, batch);
    if (s != MSOSM_OK)
        return s;
    if (!x || !logit || !offset)
        return cfail(MSOSM_ERR_BAD_ARG, "null argument");
    cudaError_t e = cudaSuccess;
    const float *xd = stage(c, x, c->xin, (size_t)batch * c->cfg.in_channels * c->cfg.length, e);
    if (e == cudaSuccess)
        e = conv_forward(c, xd, batch);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(logit, c->logit, sizeof(float) * batch, cudaMemcpyDefault, c->st);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(offset, c->off, sizeof(float) * batch, cudaMemcpyDefault, c->st);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(c->st);
    return e == cudaSuccess ? MSOSM_OK : ccuda(e, "msosm_cnn_forward");
}

msosm_status msosm_cnn_gradient(msosm_cnn *c, const float *x, const float *label, const float *target, int batch,
                                float *loss, float *grad)
{
    msosm_status s = check_batch(c, batch);
    if (s != MSOSM_OK)
        return s;
    if (!x || !label || !target)
        return cfail(MSOSM_ERR_BAD_ARG, "null argument");
    const msosm_cnn_config &g = c->cfg;
    const int L = g.length, C = g.channels, K = g.kernel;
    cudaError_t e = cudaSuccess;
    const float *xd = stage(c, x, c->xin, (size_t)batch * g.in_channels * L, e);
    const float *ld = e == cudaSuccess ? stage(c, label, c->lab, batch, e) : nullptr;
    const float *td = e == cudaSuccess ? stage(c, target, c->tgt, batch, e) : nullptr;
    if (e == cudaSuccess)
        e = conv_forward(c, xd, batch);
    if (e == cudaSuccess) {
        HeadArgs a{};
        a.h = c->h;
        a.logit = c->logit;
        a.offset = c->off;
        a.label = ld;
        a.target = td;
        a.dl = c->dl;
        a.dof = c->dof;
        a.gwd = c->grad + c->wd_off;
        a.gbd = c->grad + c->bd_off;
        a.gwr = c->grad + c->wr_off;
        a.gbr = c->grad + c->br_off;
        a.loss = c->loss;
        a.B = batch;
        a.C = C;
        a.dm_weight = g.dm_weight;
        heads_grad_kernel<<<1, kHeadThreads, 5 * sizeof(float) * kHeadThreads, c->st>>>(a);
        e = cudaGetLastError();
    }
    float *gcur = c->g0, *gnext = c->g1;
    if (e == cudaSuccess) {
        const long long n4 = (long long)batch * C * L / 4;  // at most 1024 x 256 x 256
        pool_bwd_kernel<<<nblocks(n4, 256), 256, 0, c->st>>>(
            c->dl, c->dof, c->q + c->wd_off, c->q + c->wr_off, reinterpret_cast<const float4 *>(c->act[g.layers]),
            (unsigned)C, (unsigned)L / 4, (unsigned)n4, (float)L, reinterpret_cast<float4 *>(gcur));
        e = cudaGetLastError();
    }
    WgradRows rows{};
    rows.part = c->part;
    rows.grad = c->grad;
    long long widest = 0;
    for (int l = g.layers - 1; l >= 0 && e == cudaSuccess; --l) {
        const int ci = l == 0 ? g.in_channels : C;
        const float *a_in = l == 0 ? xd : c->act[l];
        // weights and biases of a layer lie together in the gradient
        rows.offset[l] = c->part_off[l];
        rows.out[l] = c->w_off[l];
        rows.values[l] = (long long)C * ci * K + C;
        rows.groups[l] = wgrad_groups(C, ci, batch);
        widest = std::max(widest, rows.values[l]);
        e = launch_wgrad(K, gcur, C, a_in, ci, batch, L, c->part + c->part_off[l], c->st);
        if (e == cudaSuccess && l > 0) {
            e = launch_conv<true>(K, gcur, C, L, c->wb + c->w_off[l], nullptr, ci, batch, c->act[l], gnext, c->st);
            float *t = gcur;
            gcur = gnext;
            gnext = t;
        }
    }
    if (e == cudaSuccess) {
        wgrad_reduce_kernel<<<dim3((unsigned)((widest + 31) / 32), (unsigned)g.layers), 256, 0, c->st>>>(rows);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && loss)
        e = cudaMemcpyAsync(loss, c->loss, sizeof(float), cudaMemcpyDefault, c->st);
    if (e == cudaSuccess && grad)
        e = cudaMemcpyAsync(grad, c->grad, sizeof(float) * c->n, cudaMemcpyDefault, c->st);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(c->st);
    return e == cudaSuccess ? MSOSM_OK : ccuda(e, "msosm_cnn_gradient");
}

msosm_status msosm_cnn_adam_step(msosm_cnn *c, float lr)
{
    if (!c || !(lr > 0.f))
        return cfail(MSOSM_ERR_BAD_ARG, "null network or learning rate <= 0");
    c->steps += 1;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float c1 = 1.f - (float)std::pow((double)b1, (double)c->steps);
    const float c2 = 1.f - (float)std::pow((double)b2, (double)c->steps);
    adam_kernel<<<nblocks(c->n, 256), 256, 0, c->st>>>(c->th, c->grad, c->m, c->v, c->q, c->n, lr, b1, b2, c1, c2,
                                                       eps, pack_args(c));
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(c->st);
    return e == cudaSuccess ? MSOSM_OK : ccuda(e, "msosm_cnn_adam_step");
}

}  // extern "C"

// pair_dedisp.cu -- the FP32 fused dedispersion + detection + folding kernel.
//
// Persistent; per (DM trial, block range): gather each bin's delayed spectrum
// from the ring, multiply by H, inverse FFT in shared memory, keep the second
// half (overlap-save discard), then write the series and/or detect and fold.
// Replaces ComplexMultiplyDelay_concurrent_batch + inverse cufftExecC2C +
// DiscardSamples_concurrent_batch (gpu/gpu_kernel.cu:128-198,236-258) and,
// fused, the calculateIntensity kernel + host fold of Fold_GPU
// (gpu/gpu_kernel.cu:347-353, folding/fold_gpu.cpp:48-194).
//
// A thread transforms 16 points of TWO consecutive blocks of one trial at a
// time in packed FP32 (fft_pair.cuh).  At 16384 points two blocks do not fit
// in shared memory; there one radix-2 step splits a block into two 8192-point
// transforms (even and odd output samples), which run as the pair.
//
// What does not change from block to block -- the thread's filter values and
// block delays (per trial) and its stage twiddles (always) -- waits in the
// thread's tensor-memory lane, 128 columns per warp, and is read into
// registers where it is used, once per pair.
#include "fft_pair.cuh"
#include "fold_dev.cuh"
#include "kernels.hpp"
#include "tmem.cuh"

#include <cuda_runtime.h>

namespace msosm {
namespace {

using namespace pairfft;

template <int LOG2N>
struct PairShape {
    static constexpr int N = 1 << LOG2N, M = N / 2;
    static constexpr bool SPLIT = LOG2N == 14;            // one block as two half-size transforms
    static constexpr int LT = SPLIT ? LOG2N - 1 : LOG2N;  // log2 of a transform of the pair
    using F = FftShape<LT>;
    using X = PairFft<LT>;
    static constexpr int T = F::T;                        // threads per pair
    static constexpr int G = T >= 256 ? 1 : 256 / T;      // pairs per thread block
    static constexpr int THREADS = G * T;                 // 256 (512 at 8192 and 16384)
    static constexpr int CTAS_PER_SM = THREADS == 256 ? 2 : 1;
    static constexpr int BPS = SPLIT ? 1 : 2 * G;         // blocks per step
    static constexpr int STEP = BPS * M;                  // samples of a step
    static_assert(STEP == 16 * THREADS, "a step holds 16 samples per thread");
    static constexpr int IBUF = SPLIT ? kIbufPadded2 : kIbufPadded;
    static constexpr size_t SMEM_FFT = (size_t)G * X::SMEM * sizeof(float4);
    static constexpr size_t SMEM_IBUF = (size_t)ibuf_floats(STEP) * sizeof(float);
    // tensor-memory columns of one warp: filter (SPLIT: the radix-2
    // twiddles), delays, stage twiddles
    static constexpr int COL_H = 0, COL_D = 32, COLS = 128;
    __host__ __device__ static constexpr int col_stage(int s)
    {
        return s == 0 ? 48 : (s + 1 < F::NST || F::NST < 4 ? 80 : 112);
    }
    static constexpr int TMEM_COLS = COLS * (THREADS / 128);  // four warps share a lane quadrant's columns
};

template <int LOG2N, int S>
__device__ __forceinline__ void load_twiddles(float (&w)[32], uint32_t tm)
{
    using P = PairShape<LOG2N>;
    __syncwarp();  // tensor-memory reads are warp-wide
    if constexpr (P::X::words(S) <= 16) {
        uint32_t r[16];
        tmem_ld_16(tm + P::col_stage(S), r);
#pragma unroll
        for (int i = 0; i < 16; ++i)
            w[i] = __uint_as_float(r[i]);
    } else {
        uint32_t r[32];
        tmem_ld_32(tm + P::col_stage(S), r);
#pragma unroll
        for (int i = 0; i < 32; ++i)
            w[i] = __uint_as_float(r[i]);
    }
}

template <int LOG2N, int S = 0>
__device__ __forceinline__ void store_twiddles(uint32_t tm, int j, const float2 *__restrict__ tw)
{
    using P = PairShape<LOG2N>;
    if constexpr (S < P::F::NST) {
        if constexpr (P::X::words(S) > 0) {
            float w[32];
            stage_twiddles<P::LT, S, P::N>(w, j, tw);
            if constexpr (P::X::words(S) <= 16) {
                uint32_t r[16];
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    r[i] = __float_as_uint(w[i]);
                tmem_st_16(tm + P::col_stage(S), r);
            } else {
                uint32_t r[32];
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    r[i] = __float_as_uint(w[i]);
                tmem_st_32(tm + P::col_stage(S), r);
            }
        }
        store_twiddles<LOG2N, S + 1>(tm, j, tw);
    }
}

// Barrier of the T threads that share one pair's buffer.
template <int LOG2N>
__device__ __forceinline__ void pair_sync(int g)
{
    using P = PairShape<LOG2N>;
    if constexpr (P::T <= 32)
        __syncwarp();
    else if constexpr (P::G > 1)
        asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "n"(P::T) : "memory");
    else
        __syncthreads();
}

// The inverse transforms of one pair, v in register order of stage 0; the
// result in that of the last stage.  The buffer must be free on entry; on
// exit this thread has read it, but others may still be reading.
template <int LOG2N, int S = 0>
__device__ __forceinline__ void pair_ifft(c2 (&v)[16], float4 *buf, int g, int j, uint32_t tm)
{
    using P = PairShape<LOG2N>;
    constexpr int NST = P::F::NST;
    if constexpr (S > 0) {
        pair_sync<LOG2N>(g);
        stage_load<P::LT, S>(v, buf, j);
    }
    float w[32];
    if constexpr (P::X::words(S) > 0)
        load_twiddles<LOG2N, S>(w, tm);
    if constexpr (S + 1 < NST) {
        pairfft::dft16(v);
        if constexpr (P::X::words(S) > 0)
            twiddle_out(v, w);
        stage_store<P::LT, S>(v, buf, j);
        pair_ifft<LOG2N, S + 1>(v, buf, g, j, tm);
    } else {
        last_stage<P::LT>(v, w);
    }
}

template <int LOG2N, bool SERIES, bool FOLD>
__global__ void __launch_bounds__(PairShape<LOG2N>::THREADS, PairShape<LOG2N>::CTAS_PER_SM)
    pair_dedisp_kernel(const __grid_constant__ DedispArgs a)
{
    using P = PairShape<LOG2N>;
    using F = typename P::F;
    constexpr int N = P::N, M = P::M, T = P::T, BPS = P::BPS, RL = F::radix(F::NST - 1);
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int g = P::G > 1 ? tid / T : 0, j = P::G > 1 ? tid % T : tid;  // pair of the step, thread of the pair
    float4 *buf = reinterpret_cast<float4 *>(smem) + g * P::X::SMEM;
    float *ibuf = reinterpret_cast<float *>(smem + P::SMEM_FFT);
    // where this thread's first sample goes; its others are T >= 32 samples
    // on, a constant distance in the padded layout
    float *ib = ibuf + (P::SPLIT ? ipad2(2 * j) : ipad(2 * g * M + j));
    FoldSmem fw;
    if constexpr (FOLD)
        fold_smem_layout(fw, ibuf + ibuf_floats(P::STEP), a.fold);
    if (warp == 0) {
        tmem_alloc(smem_addr(&tmem_base), P::TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // this warp's lanes and columns
    const uint32_t tm = *const_cast<volatile uint32_t *>(&tmem_base) + ((uint32_t)(32 * (warp & 3)) << 16) +
                        (uint32_t)(P::COLS * (warp >> 2));
    store_twiddles<LOG2N>(tm, j, a.tw);
    if constexpr (P::SPLIT) {
        // e^{+2 pi i b / N} of the odd samples' transform, b = j + r T
        uint32_t w[32];
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const float2 x = __ldg(&a.tw[j + r * T]);
            w[2 * r] = __float_as_uint(x.x);
            w[2 * r + 1] = __float_as_uint(x.y);
        }
        tmem_st_32(tm + P::COL_H, w);
    }
    const int smask = a.S - 1;  // the ring depth is a power of two
    // a ring of up to 4 GB is addressed with 32-bit byte offsets
    const bool small_ring = (unsigned long long)a.S * N * sizeof(float2) <= 1ull << 32;
    const uint32_t bmask = (uint32_t)((unsigned long long)a.S * N * sizeof(float2) - 1);
    const int items = a.D * a.R;
    const int nunits = (a.count + BPS - 1) / BPS;  // steps of the whole call
    // items beyond the first are handed out from a counter: the CTAs of the
    // two dies and of SMs with one or two resident CTAs do not run equally fast,
    // and with a fixed stride an eighth of the CTA slots stood empty at the end.
    // The next item is fetched while this one runs.
    __shared__ int next_item;
    int w = blockIdx.x;
    while (w < items) {
        if (tid == 0)
            next_item = (int)gridDim.x + atomicAdd(&a.work[0], 1);
        const int dm = w % a.D;
        const int rr = w / a.D;
        const int kb = BPS * (int)((long long)nunits * rr / a.R);
        const int ke = min(a.count, BPS * (int)((long long)nunits * (rr + 1) / a.R));
        const float2 *__restrict__ Hd = a.H + (size_t)dm * N + j;
        const uint16_t *__restrict__ dl = a.delays + (size_t)dm * N + j;
        if constexpr (!P::SPLIT) {
            uint32_t h[32], d[16];
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                const float2 x = __ldg(Hd + r * T);
                h[2 * r] = __float_as_uint(x.x);
                h[2 * r + 1] = __float_as_uint(x.y);
                // byte offset of bin b, its block delay back: wraps mod the ring
                d[r] = (uint32_t)(j + r * T - (int)__ldg(dl + r * T) * N) * (uint32_t)sizeof(float2);
            }
            __syncwarp();
            tmem_st_32(tm + P::COL_H, h);
            tmem_st_16(tm + P::COL_D, d);
        } else {
            // the block delays of bins j + r T and M further, one word
            uint32_t d[16];
#pragma unroll
            for (int r = 0; r < 16; ++r)
                d[r] = (uint32_t)__ldg(dl + r * T) | (uint32_t)__ldg(dl + M + r * T) << 16;
            __syncwarp();
            tmem_st_16(tm + P::COL_D, d);
        }
        FoldCursor cursor;
        if constexpr (FOLD) {
            if (a.fold.smem_prof) {
                for (int i = tid; i < 2 * a.fold.nbins; i += P::THREADS)
                    fw.prof_main[i] = 0.f;
            } else {
                fw.prof_main = a.fold.part_main + (size_t)w * a.fold.nbins;
                fw.prof_pend = a.fold.part_pend + (size_t)w * a.fold.nbins;
            }
            cursor_init(a.fold, fw, cursor, (long long)kb * M);
        }
        // the delayed spectra of the pair at block k + 2 g, this thread's bins:
        // blocks k, k + 1 at bin j + r T; SPLIT: block k at bins j + r T and
        // M further
        float2 xa[16], xb[16];
        auto gather = [&](int k) {
            const int k0 = k + (P::SPLIT ? 0 : 2 * g);
            const long long kg = a.k0 + k0;
            const int slot = (int)(kg & smask);
            const float2 *__restrict__ base = a.ring + j;
            __syncwarp();
            if constexpr (!P::SPLIT) {
                const bool two = k0 + 1 < ke;
                if (__all_sync(0xffffffffu, kg >= a.max_delay && two) && small_ring) {
                    // every delayed block exists: byte offsets in the ring as
                    // 32-bit sums, wrapped by a mask
                    uint32_t e[16];
                    tmem_ld_16(tm + P::COL_D, e);
                    const uint32_t s0 = (uint32_t)slot * (uint32_t)(N * sizeof(float2)), s1 = s0 + (uint32_t)(N * sizeof(float2));
                    const char *ring = reinterpret_cast<const char *>(a.ring);
#pragma unroll
                    for (int r = 0; r < 16; ++r) {
                        xa[r] = *reinterpret_cast<const float2 *>(ring + ((s0 + e[r]) & bmask));
                        xb[r] = *reinterpret_cast<const float2 *>(ring + ((s1 + e[r]) & bmask));
                    }
                } else {
#pragma unroll
                    for (int r = 0; r < 16; ++r) {
                        const int d = __ldg(dl + r * T);
                        xa[r] = xb[r] = make_float2(0.f, 0.f);
                        // blocks before the stream start are zero, and so are
                        // the missing blocks of the call's last step
                        if (k0 < ke && kg >= d)
                            xa[r] = base[(size_t)((slot - d) & smask) * N + r * T];
                        if (two && kg + 1 >= d)
                            xb[r] = base[(size_t)((slot - d + 1) & smask) * N + r * T];
                    }
                }
            } else if (kg >= a.max_delay && small_ring) {
                uint32_t d[16];
                tmem_ld_16(tm + P::COL_D, d);
                const char *ring = reinterpret_cast<const char *>(a.ring + j);
#pragma unroll
                for (int r = 0; r < 16; ++r) {
                    constexpr uint32_t ROW = (uint32_t)(N * sizeof(float2));
                    const uint32_t o0 = (uint32_t)((slot - (int)(d[r] & 0xFFFFu)) & smask) * ROW;
                    const uint32_t o1 = (uint32_t)((slot - (int)(d[r] >> 16)) & smask) * ROW;
                    xa[r] = reinterpret_cast<const float2 *>(ring + o0)[r * T];
                    xb[r] = reinterpret_cast<const float2 *>(ring + o1)[M + r * T];
                }
            } else {
#pragma unroll
                for (int r = 0; r < 16; ++r) {
                    const int d0 = __ldg(dl + r * T), d1 = __ldg(dl + M + r * T);
                    xa[r] = xb[r] = make_float2(0.f, 0.f);
                    if (kg >= d0)
                        xa[r] = base[(size_t)((slot - d0) & smask) * N + r * T];
                    if (kg >= d1)
                        xb[r] = base[(size_t)((slot - d1) & smask) * N + M + r * T];
                }
            }
        };
        for (int k = kb; k < ke; k += BPS) {
            gather(k);
            const int k0 = k + (P::SPLIT ? 0 : 2 * g);  // this pair's first block
            c2 v[16];
            __syncwarp();  // the tensor-memory reads below are warp-wide
            if constexpr (!P::SPLIT) {
                uint32_t h[32];
                tmem_ld_32(tm + P::COL_H, h);
#pragma unroll
                for (int r = 0; r < 16; ++r) {
                    const float2 hv = make_float2(__uint_as_float(h[2 * r]), __uint_as_float(h[2 * r + 1]));
                    const float2 za = cmul(xa[r], hv), zb = cmul(xb[r], hv);
                    v[r] = {pk(za.x, zb.x), pk(za.y, zb.y)};
                }
            } else {
                // Z[b] +- Z[b + N/2], the difference times e^{2 pi i b / N}
                uint32_t t[32];
                tmem_ld_32(tm + P::COL_H, t);
#pragma unroll
                for (int r = 0; r < 16; ++r) {
                    const float2 za = cmul(xa[r], __ldg(Hd + r * T)), zb = cmul(xb[r], __ldg(Hd + M + r * T));
                    const float2 s = ::msosm::cadd(za, zb);
                    const float2 o = cmul(::msosm::csub(za, zb),
                                          make_float2(__uint_as_float(t[2 * r]), __uint_as_float(t[2 * r + 1])));
                    v[r] = {pk(s.x, o.x), pk(s.y, o.y)};
                }
            }
            // every thread has read the previous step's last stage: with
            // folding the barrier ahead of the fold sees to that
            if constexpr (!FOLD)
                pair_sync<LOG2N>(g);
            pair_ifft<LOG2N>(v, buf, g, j, tm);
            // pairs that do not take part in each other's barriers: the
            // previous step's fold has read the intensities
            if constexpr (FOLD && P::G > 1)
                __syncthreads();
            // keep outputs n >= half (the last-stage slots with r >= R/2)
#pragma unroll
            for (int slot_ = 0; slot_ < 16; ++slot_) {
                if ((slot_ % RL) >= RL / 2) {
                    const int t = last_out_index<P::LT>(j, slot_) - F::N / 2;
                    const float2 re = upk(v[slot_].re), im = upk(v[slot_].im);
                    if constexpr (SERIES) {
                        float2 *out = a.series + (size_t)dm * a.count * M + (size_t)k0 * M;
                        if constexpr (P::SPLIT) {
                            *reinterpret_cast<float4 *>(out + 2 * t) = make_float4(re.x, im.x, re.y, im.y);
                        } else {
                            if (k0 < ke)
                                out[t] = make_float2(re.x, im.x);
                            if (k0 + 1 < ke)
                                out[M + t] = make_float2(re.y, im.y);
                        }
                    }
                    if constexpr (FOLD) {
                        const f2 p2 = fma2(v[slot_].re, v[slot_].re, mul2(v[slot_].im, v[slot_].im));
                        float2 p = upk(p2);
                        if (a.fold.detect)
                            p = make_float2(sqrtf(p.x), sqrtf(p.y));
                        if constexpr (P::SPLIT) {
                            // samples 2t and 2t + 1
                            *reinterpret_cast<float2 *>(ib + ipad2(2 * (t - j))) = p;
                        } else if constexpr (T >= 32) {
                            ib[ipad(t - j)] = p.x;
                            ib[ipad(M + t - j)] = p.y;
                        } else {
                            ibuf[ipad(2 * g * M + t)] = p.x;
                            ibuf[ipad((2 * g + 1) * M + t)] = p.y;
                        }
                    }
                }
            }
            if constexpr (FOLD)
                __syncthreads();
            if constexpr (FOLD)
                fold_block<P::IBUF>(a.fold, fw, ibuf, k * M, min(ke - k, BPS) * M, cursor, 160 * ((k / BPS) & 15));
        }
        if constexpr (FOLD) {
            __syncthreads();
            if (a.fold.smem_prof) {
                float *gm = a.fold.part_main + (size_t)w * a.fold.nbins;
                float *gp = a.fold.part_pend + (size_t)w * a.fold.nbins;
                for (int i = tid; i < a.fold.nbins; i += P::THREADS) {
                    gm[i] = fw.prof_main[i];
                    if (rr >= a.fold.pend_row)
                        gp[i] = fw.prof_pend[i];
                }
            }
        }
        __syncthreads();
        w = next_item;
        __syncthreads();
    }
    // the last CTA to finish leaves the counter at zero for the next launch
    if (tid == 0 && atomicAdd(&a.work[1], 1) == (int)gridDim.x - 1) {
        a.work[0] = 0;
        a.work[1] = 0;
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(*const_cast<volatile uint32_t *>(&tmem_base), P::TMEM_COLS);
    }
}

// Calls go(kernel) with the instantiation for (series, fold).
template <int LOG2N, typename G>
auto pair_select(bool series, bool fold, G &&go)
{
    if (series && fold)
        return go(pair_dedisp_kernel<LOG2N, true, true>);
    if (fold)
        return go(pair_dedisp_kernel<LOG2N, false, true>);
    return go(pair_dedisp_kernel<LOG2N, true, false>);
}

template <int LOG2N>
size_t pair_smem(bool fold, size_t fold_smem)
{
    using P = PairShape<LOG2N>;
    return P::SMEM_FFT + (fold ? P::SMEM_IBUF + fold_smem : 0);
}

template <int LOG2N>
cudaError_t launch_t(bool series, bool fold, const DedispArgs &a, int grid, cudaStream_t st)
{
    using P = PairShape<LOG2N>;
    const size_t sm = pair_smem<LOG2N>(
        fold, fold ? fold_smem_bytes(a.fold.nbins, a.fold.span_cap, a.fold.smem_prof != 0) : 0);
    return pair_select<LOG2N>(series, fold, [&](auto k) -> cudaError_t {
        cudaError_t e = allow_smem(k, sm);
        if (e != cudaSuccess)
            return e;
        k<<<grid, P::THREADS, sm, st>>>(a);
        return cudaGetLastError();
    });
}

}  // namespace

#define MSOSM_PAIR_DISPATCH(log2n, CALL)                                                                               \
    switch (log2n) {                                                                                                   \
    case 6: return CALL(6);                                                                                            \
    case 7: return CALL(7);                                                                                            \
    case 8: return CALL(8);                                                                                            \
    case 9: return CALL(9);                                                                                            \
    case 10: return CALL(10);                                                                                          \
    case 11: return CALL(11);                                                                                          \
    case 12: return CALL(12);                                                                                          \
    case 13: return CALL(13);                                                                                          \
    case 14: return CALL(14);                                                                                          \
    default: break;                                                                                                    \
    }

cudaError_t launch_dedisp(int log2n, bool series, bool fold, const DedispArgs &a, int grid, cudaStream_t st)
{
    if (!series && !fold)
        return cudaErrorInvalidValue;
#define CALL(L) launch_t<L>(series, fold, a, grid, st)
    MSOSM_PAIR_DISPATCH(log2n, CALL)
#undef CALL
    return cudaErrorInvalidValue;
}

int dedisp_blocks_per_step(int log2n)
{
#define CALL(L) PairShape<L>::BPS
    MSOSM_PAIR_DISPATCH(log2n, CALL)
#undef CALL
    return 1;
}

size_t dedisp_smem(int log2n, bool fold, size_t fold_smem)
{
#define CALL(L) pair_smem<L>(fold, fold_smem)
    MSOSM_PAIR_DISPATCH(log2n, CALL)
#undef CALL
    return 0;
}

// Dynamic shared memory one CTA may use while all the CTAs the kernel is
// built for stay resident (64 bytes left for its static variables).
size_t dedisp_smem_share(int log2n)
{
    int dev = 0, sm = 0, block = 0, reserved = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&block, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev) != cudaSuccess)
        return 0;
    const int share = sm / dedisp_ctas_per_sm(log2n) - reserved;
    return (size_t)((share < block ? share : block) - 64);
}

int dedisp_ctas_per_sm(int log2n) { return log2n >= 13 ? PairShape<13>::CTAS_PER_SM : PairShape<12>::CTAS_PER_SM; }

}  // namespace msosm

// kernels.cu -- sm_100a kernels of the MS-OSM / OSM dedispersion path (the
// fused dedispersion kernels are in pair_dedisp.cu and tc_dedisp.cu).
//
//   forward_kernel  decode (uint16 offset-binary or complex64) + forward FFT of
//                   the overlapping windows of one call, written into the
//                   spectrum ring shared by all DM trials.  Replaces
//                   uint16ToComplex + the forward cufftExecC2C
//                   (gpu/gpu_kernel.cu:276-299, msosm_gpu_dm_concurrent.cpp:123-129).
//   design_kernel   dedispersion filter H per trial on the device: FP64 chirp
//                   phase reduced mod 2 pi, M-point inverse FFT, zero pad,
//                   2M-point FFT (msosm_prepare.cpp:37-84 on the host in the
//                   reference).
//
// Ring semantics: the reference scatters X[c][b]*H[b]/N into a per-DM product
// ring at slot (index + c + delay[b]) % S and inverse-transforms slots
// index..index+count-1 (gpu/gpu_kernel.cu:179-184).  A slot therefore holds,
// for bin b, the product of block k - delay[b] (zero before the stream
// start).  Here the ring holds the input spectra once for all trials and
// each trial gathers X[k - delay[b]][b] * H[b] directly.
#include "chirp.cuh"
#include "fft_smem.cuh"
#include "kernels.hpp"
#include "tc_layout.hpp"

#include <algorithm>
#include <map>
#include <mutex>
#include <utility>

#include <cuda.h>
#include <cuda_runtime.h>

namespace msosm {

// ---------------------------------------------------------------------------
// forward transform of the input windows
// ---------------------------------------------------------------------------

template <int KIND>
__device__ __forceinline__ float2 load_sample(const void *p, long long s)
{
    if constexpr (KIND == kInputC64) {
        return reinterpret_cast<const float2 *>(p)[s];
    } else {
        // offset binary, 0 = blank (gpu/gpu_kernel.cu:291-296)
        const uint32_t u = reinterpret_cast<const uint32_t *>(p)[s];
        const uint32_t x = u & 0xFFFFu, y = u >> 16;
        return make_float2(x ? (float)x - 32768.0f : 0.0f, y ? (float)y - 32768.0f : 0.0f);
    }
}

template <int LOG2N, int KIND, bool PP>
__global__ void __launch_bounds__(FftShape<LOG2N>::T) forward_kernel(FwdArgs a)
{
    using F = FftShape<LOG2N>;
    constexpr int N = F::N, M = N / 2, T = F::T;
    extern __shared__ float2 smem[];
    float2 *buf0 = smem;
    float2 *buf1 = PP ? smem + F::SMEM : smem;
    const int tid = threadIdx.x;
    const int c = blockIdx.x;
    float2 v[16];
    // window c covers input samples [c*M - M, c*M + M); negative indices are
    // the previous call's last M samples (the reference's D2D overlap copy,
    // msosm_gpu_dm_concurrent.cpp:125)
#pragma unroll
    for (int r = 0; r < 16; ++r) {
        const int n = tid + r * T;
        const long long s = (long long)c * M + n - M;
        const float2 x = (s < 0) ? a.hist_in[M + s] : load_sample<KIND>(a.input, s);
        if (c == a.count - 1 && n >= M)
            a.hist_out[n - M] = x;
        v[r] = x;
    }
    dft16<-1>(v);
    stage_store<LOG2N, 0>(v, buf0, tid);
    run_stages<LOG2N, -1, PP>(v, buf0, buf1, tid, a.tw);
    const int slot_row = (int)((a.k0 + c) & (a.S - 1));
    float2 *row = a.ring + (size_t)slot_row * N;
    if ((LOG2N >= 12 && LOG2N <= 14) && a.tc_order) {
        float mx = 0.f;
#pragma unroll
        for (int slot = 0; slot < 16; ++slot) {
            row[tc::tc_pos(last_out_index<LOG2N>(tid, slot), LOG2N)] = v[slot];
            mx = fmaxf(mx, fmaxf(fabsf(v[slot].x), fabsf(v[slot].y)));
        }
        // the row's largest component (the tensor-core kernel scales by it)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        __syncthreads();  // every thread is done with the FFT buffers
        float *wm = reinterpret_cast<float *>(buf0);
        if ((tid & 31) == 0)
            wm[tid >> 5] = mx;
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < T / 32; ++w)
                mx = fmaxf(mx, wm[w]);
            a.row_max[slot_row] = mx;
        }
    } else {
#pragma unroll
        for (int slot = 0; slot < 16; ++slot)
            row[last_out_index<LOG2N>(tid, slot)] = v[slot];
    }
}

// ---------------------------------------------------------------------------
// folding of a materialised intensity series (Fold_GPU)
// ---------------------------------------------------------------------------

// sqrt(|a|^2 + |b|^2) per sample (b may be null): gpu/gpu_kernel.cu:347-353.
__global__ void intensity_kernel(const float2 *__restrict__ a, const float2 *__restrict__ b, float *__restrict__ out,
                                 size_t n)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const float2 x = a[i];
        float p = x.x * x.x + x.y * x.y;
        if (b) {
            const float2 y = b[i];
            p += y.x * y.x + y.y * y.y;
        }
        out[i] = sqrtf(p);
    }
}

// Fold the intensities of a chunk straight from memory: a group of G = 2^g_shift
// lanes per output bin adds the bin's samples of every span of row r's share
// [nspans r / R, nspans (r + 1) / R) and writes them to partial row r (the main
// and the pending sums); trial d = blockIdx.z folds I[d n ...] into rows r D + d.
// For bins of up to 1024 samples, and up to 4096 where the chunk fills a
// thousand of them (fold_wide): a lane adds at most 128 samples of a span (32
// to an accumulator) and eight spans in FP32, more spans in FP64.
// Bound by latency: a lane's loads are independent, and blocks and rows are
// cut so that about 1200 blocks share the chunk (fold_direct_rows).  At 84
// periods of 49600 samples and 1024 bins the staged form (2048 samples to
// shared memory, then folded by the block, 592 rows) took 26 us.
__global__ void __launch_bounds__(256) fold_direct_kernel(const float *__restrict__ I, long long n, FoldArgs f)
{
    const int r = blockIdx.y, R = gridDim.y, d = blockIdx.z, D = gridDim.z;
    I += (size_t)d * n;
    const int G = 1 << f.g_shift, l = threadIdx.x & (G - 1);
    const int bin = (int)blockIdx.x * (256 >> f.g_shift) + (int)(threadIdx.x >> f.g_shift);
    const int s0 = (int)((long long)f.nspans * r / R), s1 = (int)((long long)f.nspans * (r + 1) / R);
    // the sums of eight spans in FP32, more in FP64
    const bool many = s1 - s0 > 8, with_pend = r >= f.pend_row;
    float main = 0.f, pend = 0.f;
    double mains = 0.0, pends = 0.0;
    if (bin < f.nbins) {
        const long long p0 = (long long)bin * f.bpt;
        for (int s = s0; s < s1; ++s) {
            if (many && ((s - s0) & 7) == 0) {
                mains += (double)main;
                pends += (double)pend;
                main = pend = 0.f;
            }
            const int dest = f.span_dest[s];
            if (dest == 0)
                continue;
            const long long a = f.span_a[s], ph = f.span_phase0[s], len = f.span_b[s] - a;
            const long long lo = p0 > ph ? p0 : ph, hi = p0 + f.bpt < ph + len ? p0 + f.bpt : ph + len;
            const float *src = I + (a - ph) + lo;  // (only read below hi)
            const int m = hi > lo ? (int)(hi - lo) : 0;
            float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
            int p = l;
            for (; p + 3 * G < m; p += 4 * G) {
                a0 += src[p];
                a1 += src[p + G];
                a2 += src[p + 2 * G];
                a3 += src[p + 3 * G];
            }
            if (p < m)
                a0 += src[p];
            if (p + G < m)
                a1 += src[p + G];
            if (p + 2 * G < m)
                a2 += src[p + 2 * G];
            const float sum = (a0 + a1) + (a2 + a3);
            if (dest == 1)
                main += sum;
            else
                pend += sum;
        }
    }
    if (many) {
        mains += (double)main;
        pends += (double)pend;
        for (int o = G >> 1; o > 0; o >>= 1) {
            mains += __shfl_xor_sync(0xffffffffu, mains, o);
            if (with_pend)
                pends += __shfl_xor_sync(0xffffffffu, pends, o);
        }
        main = (float)mains;
        pend = (float)pends;
    } else {
        for (int o = G >> 1; o > 0; o >>= 1) {
            main += __shfl_xor_sync(0xffffffffu, main, o);
            if (with_pend)
                pend += __shfl_xor_sync(0xffffffffu, pend, o);
        }
    }
    if (bin < f.nbins && l == 0) {
        const size_t at = ((size_t)r * D + d) * f.nbins + bin;
        f.part_main[at] = main;
        if (with_pend)
            f.part_pend[at] = pend;
    }
}

// The same for long bins (fold_wide): partial row r takes the samples
// [n r / R, n (r + 1) / R) whatever spans they lie in, and the whole
// block adds the samples of a bin.  With few long bins the form above has
// nothing to share out: at 4 bins of 2.8 million samples one span's worth of
// lanes did everything, 2.4 ms a call of 2^20 samples (37 us here, of which 35 are
// the call and its readout).
// A thread adds at most 64 samples in FP32 (16 to an accumulator); those sums,
// the threads and the spans in FP64.
// A row shorter than a period touches the bins from that of its first sample
// on, at most len / bpt + 3 of them; the others are zero.
__global__ void __launch_bounds__(256) fold_wide_kernel(const float *__restrict__ I, long long n, FoldArgs f)
{
    constexpr int W = 8, GROUP = 16;  // warps; bins between two barriers
    __shared__ double sums[2][GROUP][W];
    const int r = blockIdx.x, R = gridDim.x, d = blockIdx.y, D = gridDim.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long t0 = n * r / R, t1 = n * (r + 1) / R;
    I += (size_t)d * n;
    const size_t row = ((size_t)r * D + d) * f.nbins;
    const bool with_pend = r >= f.pend_row;
    for (int i = threadIdx.x; i < f.nbins; i += 256) {
        f.part_main[row + i] = 0.f;
        if (with_pend)
            f.part_pend[row + i] = 0.f;
    }
    // the spans that reach into the row
    int lo = 0, s1 = f.nspans;
    while (lo < s1) {
        const int mid = (lo + s1) >> 1;
        if (f.span_b[mid] <= t0)
            lo = mid + 1;
        else
            s1 = mid;
    }
    const int s0 = lo;
    if (s0 >= f.nspans || f.span_a[s0] >= t1)
        return;
    for (s1 = s0 + 1; s1 < f.nspans && f.span_a[s1] < t1;)
        ++s1;
    const long long a0 = f.span_a[s0];
    const long long first = (f.span_phase0[s0] + (t0 > a0 ? t0 - a0 : 0)) / f.bpt;
    const long long most = (t1 - t0) / f.bpt + 3;
    const int b0 = first < f.nbins ? (int)first : 0, count = most < f.nbins ? (int)most : f.nbins;
    for (int c0 = 0; c0 < count; c0 += GROUP) {
        const int cn = min(GROUP, count - c0);
        __syncthreads();  // the zeroes are written, the last group's sums read
        for (int c = 0; c < cn; ++c) {
            int bin = b0 + c0 + c;
            bin -= bin >= f.nbins ? f.nbins : 0;
            const long long p0 = (long long)bin * f.bpt;
            double main = 0.0, pend = 0.0;
            for (int s = s0; s < s1; ++s) {
                const int dest = f.span_dest[s];
                if (dest == 0)
                    continue;
                // samples [x, y) of the chunk: this bin, this span, this row
                const long long off = f.span_a[s] - f.span_phase0[s];
                const long long x = max(max(f.span_a[s], t0), off + p0);
                const long long y = min(min(f.span_b[s], t1), off + p0 + f.bpt);
                double sum = 0.0;
                for (long long q = x; q < y; q += 64 * 256) {
                    const int m = (int)min(y - q, 64ll * 256);
                    const float *src = I + q;
                    float v0 = 0.f, v1 = 0.f, v2 = 0.f, v3 = 0.f;
                    int p = threadIdx.x;
                    for (; p + 3 * 256 < m; p += 4 * 256) {
                        v0 += src[p];
                        v1 += src[p + 256];
                        v2 += src[p + 2 * 256];
                        v3 += src[p + 3 * 256];
                    }
                    if (p < m)
                        v0 += src[p];
                    if (p + 256 < m)
                        v1 += src[p + 256];
                    if (p + 2 * 256 < m)
                        v2 += src[p + 2 * 256];
                    sum += (double)((v0 + v1) + (v2 + v3));
                }
                if (dest == 1)
                    main += sum;
                else
                    pend += sum;
            }
            for (int o = 16; o > 0; o >>= 1) {
                main += __shfl_xor_sync(0xffffffffu, main, o);
                pend += __shfl_xor_sync(0xffffffffu, pend, o);
            }
            if (lane == 0) {
                sums[0][c][warp] = main;
                sums[1][c][warp] = pend;
            }
        }
        __syncthreads();
        const int c = threadIdx.x >> 1, which = threadIdx.x & 1;
        if (c < cn && (which == 0 || with_pend)) {
            double v = 0.0;
#pragma unroll
            for (int w = 0; w < W; ++w)
                v += sums[which][c][w];
            int bin = b0 + c0 + c;
            bin -= bin >= f.nbins ? f.nbins : 0;
            (which ? f.part_pend : f.part_main)[row + bin] = (float)v;
        }
    }
}

// ---------------------------------------------------------------------------
// filter design on the device
// ---------------------------------------------------------------------------

template <int LOG2N, bool PP>
__global__ void __launch_bounds__(FftShape<LOG2N>::T) design_kernel(DesignArgs a)
{
    using F = FftShape<LOG2N>;
    using FM = FftShape<LOG2N - 1>;
    constexpr int N = F::N, M = N / 2, T = F::T, TM = FM::T;
    extern __shared__ float2 smem[];
    float2 *buf0 = smem;
    float2 *buf1 = PP ? smem + F::SMEM : smem;
    const int tid = threadIdx.x;
    const int dm = blockIdx.x;
    const ChirpParams cp = a.chirp[dm];
    const bool act = tid < TM;
    float2 v[16];
    if (act) {
        // h index j holds offset index (j + M/2) mod M (msosm_prepare.cpp:50-63)
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const int j = tid + r * TM;
            const unsigned int i = (unsigned int)((j + M / 2) & (M - 1));
            float c, s;
            chirp_cis(chirp_phase(cp, i), c, s);
            v[r] = make_float2(c, a.sign < 0 ? -s : s);
        }
        dft16<+1>(v);
        stage_store<LOG2N - 1, 0>(v, buf0, tid);
    }
    run_stages<LOG2N - 1, +1, PP>(v, buf0, buf1, tid, a.tw_inv_m, act);
    __syncthreads();
    if (act) {
#pragma unroll
        for (int slot = 0; slot < 16; ++slot)
            buf1[smem_pad(last_out_index<LOG2N - 1>(tid, slot))] = v[slot];
    }
    __syncthreads();
    // zero-padded 2M-point forward transform of the M-point result
#pragma unroll
    for (int r = 0; r < 16; ++r) {
        const int n = tid + r * T;
        v[r] = n < M ? buf1[smem_pad(n)] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    dft16<-1>(v);
    stage_store<LOG2N, 0>(v, buf0, tid);
    run_stages<LOG2N, -1, PP>(v, buf0, buf1, tid, a.tw_fwd_n);
    float2 *out = a.H + (size_t)dm * N;
#pragma unroll
    for (int slot = 0; slot < 16; ++slot) {
        const float2 y = v[slot];
        out[last_out_index<LOG2N>(tid, slot)] = make_float2(y.x * a.scale, y.y * a.scale);
    }
}

// ---------------------------------------------------------------------------
// small kernels
// ---------------------------------------------------------------------------

// Sum of the R partial rows of every (trial, bin), in double and in a fixed
// order: G groups of rows (group g: rows g, g + G, ...) are summed by G
// threads, then thread g = 0 adds the G group sums in group order.  The
// pending rows before pend_row hold nothing.  After a timed-out kernel (status
// set) the rows are incomplete and nothing is added.
// A thread block covers 32 consecutive (trial, bin) indices x G groups; row r
// of index i sits at r * D * nbins + i, so a warp reads 128 contiguous bytes of
// a row.
template <int G>
__global__ void __launch_bounds__(32 * G) fold_reduce_kernel(const float *__restrict__ pm,
                                                             const float *__restrict__ pp, long long n, int R,
                                                             int pend_row, const int *__restrict__ status, double *am,
                                                             double *ap)
{
    __shared__ double part[2][G][32];
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
    const long long i = (long long)blockIdx.x * 32 + lane;
    const bool skip = status && *status != 0;
    double sm = 0.0, sp = 0.0;
    if (i < n && !skip) {
#pragma unroll 4
        for (int r = g; r < R; r += G)
            sm += (double)pm[(size_t)r * (size_t)n + (size_t)i];
        for (int r = pend_row + g; r < R; r += G)
            sp += (double)pp[(size_t)r * (size_t)n + (size_t)i];
    }
    part[0][g][lane] = sm;
    part[1][g][lane] = sp;
    __syncthreads();
    if (g == 0 && i < n && !skip) {
        double a = 0.0, b = 0.0;
#pragma unroll
        for (int k = 0; k < G; ++k) {
            a += part[0][k][lane];
            b += part[1][k][lane];
        }
        am[i] += a;
        ap[i] += b;
    }
}

// The same for many (trial, bin) indices, four to a lane as one 16-byte read
// (n a multiple of 4), eight groups of rows: 128 trials x 1024 bins x 16 rows,
// 8.4 MB, at the memory's rate (63 us in the form above with the pending rows
// read as well).
__global__ void __launch_bounds__(256) fold_reduce4_kernel(const float4 *__restrict__ pm,
                                                           const float4 *__restrict__ pp, long long n4, int R,
                                                           int pend_row, const int *__restrict__ status,
                                                           double *__restrict__ am, double *__restrict__ ap)
{
    constexpr int G = 8;
    __shared__ double part[G][32][4];
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
    const long long i = (long long)blockIdx.x * 32 + lane;
    if (status && *status != 0)
        return;
    auto sum = [&](const float4 *rows, int r0, double *acc) {
        double s[4] = {0.0, 0.0, 0.0, 0.0};
        if (i < n4)
#pragma unroll 4
            for (int r = r0 + g; r < R; r += G) {
                const float4 v = rows[(size_t)r * (size_t)n4 + (size_t)i];
                s[0] += (double)v.x;
                s[1] += (double)v.y;
                s[2] += (double)v.z;
                s[3] += (double)v.w;
            }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4; ++k)
            part[g][lane][k] = s[k];
        __syncthreads();
        // 128 threads add the groups, one value each
        const int t = threadIdx.x;
        const long long at = (long long)blockIdx.x * 128 + t;
        if (t < 128 && at < 4 * n4) {
            double a = 0.0;
#pragma unroll
            for (int k = 0; k < G; ++k)
                a += part[k][t >> 2][t & 3];
            acc[at] += a;
        }
    };
    sum(pm, 0, am);
    if (pend_row < R)  // uniform
        sum(pp, pend_row, ap);
}

__global__ void fold_flush_kernel(double *am, double *ap, size_t n)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        am[i] += ap[i];
        ap[i] = 0.0;
    }
}

__global__ void fold_readout_kernel(const double *am, size_t n, double scale, float *out)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        out[i] = (float)(am[i] * scale);
}

// complexToUint16 (gpu/gpu_kernel.cu:317-329): uint16(v + 32768*(v != 0)),
// truncating; out-of-range values saturate (undefined in the reference).
__device__ __forceinline__ uint32_t encode_u16(float v)
{
    float u = v + (v != 0.0f ? 32768.0f : 0.0f);
    u = fminf(fmaxf(u, 0.0f), 65535.0f);
    return (uint32_t)u;
}

__global__ void encode_u16_kernel(const float2 *__restrict__ src, uint32_t *__restrict__ dst, size_t n)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const float2 v = src[i];
        dst[i] = encode_u16(v.x) | (encode_u16(v.y) << 16);
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------

bool log2n_supported(int log2n) { return log2n >= kMinLog2N && log2n <= kMaxLog2N; }

template <int LOG2N>
constexpr bool use_pingpong() { return LOG2N <= 12; }

template <int LOG2N>
size_t fft_smem_bytes()
{
    using F = FftShape<LOG2N>;
    return (use_pingpong<LOG2N>() ? 2 : 1) * F::SMEM * sizeof(float2);
}

unsigned long long context_id()
{
    using GetId = CUresult (*)(CUcontext, unsigned long long *);
    static const GetId get = [] {
        void *f = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault) != cudaSuccess)
            cudaGetLastError();
        return reinterpret_cast<GetId>(f);
    }();
    unsigned long long id = 0;
    return get && get(nullptr, &id) == CUDA_SUCCESS ? id : 0;
}

cudaError_t allow_smem(const void *kernel, size_t bytes, bool max_carveout)
{
    static std::mutex m;
    static std::map<std::pair<const void *, unsigned long long>, size_t> allowed;
    const unsigned long long ctx = context_id();
    const std::lock_guard<std::mutex> lock(m);
    if (ctx) {
        const auto it = allowed.find({kernel, ctx});
        if (it != allowed.end() && it->second >= bytes)
            return cudaSuccess;
    }
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess && max_carveout)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess && ctx)
        allowed[{kernel, ctx}] = bytes;
    return e;
}

template <int LOG2N>
static cudaError_t forward_t(InputKind kind, const FwdArgs &a, cudaStream_t st)
{
    constexpr bool PP = use_pingpong<LOG2N>();
    const size_t sm = fft_smem_bytes<LOG2N>();
    cudaError_t e;
    if (kind == kInputU16) {
        auto k = forward_kernel<LOG2N, kInputU16, PP>;
        if ((e = allow_smem(k, sm)) != cudaSuccess)
            return e;
        k<<<a.count, FftShape<LOG2N>::T, sm, st>>>(a);
    } else {
        auto k = forward_kernel<LOG2N, kInputC64, PP>;
        if ((e = allow_smem(k, sm)) != cudaSuccess)
            return e;
        k<<<a.count, FftShape<LOG2N>::T, sm, st>>>(a);
    }
    return cudaGetLastError();
}

size_t fold_smem_bytes(int nbins, int span_cap, bool smem_prof)
{
    return (size_t)span_cap * 4 * sizeof(int) + (smem_prof ? 2 * (size_t)nbins * sizeof(float) : 0);
}

template <int LOG2N>
static cudaError_t design_t(const DesignArgs &a, cudaStream_t st)
{
    constexpr bool PP = use_pingpong<LOG2N>();
    const size_t sm = fft_smem_bytes<LOG2N>();
    auto k = design_kernel<LOG2N, PP>;
    cudaError_t e = allow_smem(k, sm);
    if (e != cudaSuccess)
        return e;
    k<<<a.D, FftShape<LOG2N>::T, sm, st>>>(a);
    return cudaGetLastError();
}

#define MSOSM_DISPATCH(log2n, CALL)                                                                   \
    switch (log2n) {                                                                                  \
    case 6: return CALL(6);                                                                           \
    case 7: return CALL(7);                                                                           \
    case 8: return CALL(8);                                                                           \
    case 9: return CALL(9);                                                                           \
    case 10: return CALL(10);                                                                         \
    case 11: return CALL(11);                                                                         \
    case 12: return CALL(12);                                                                         \
    case 13: return CALL(13);                                                                         \
    case 14: return CALL(14);                                                                         \
    default: break;                                                                                   \
    }

cudaError_t launch_forward(int log2n, InputKind kind, const FwdArgs &a, cudaStream_t st)
{
#define CALL(L) forward_t<L>(kind, a, st)
    MSOSM_DISPATCH(log2n, CALL)
#undef CALL
    return cudaErrorInvalidValue;
}

cudaError_t launch_design(int log2n, const DesignArgs &a, cudaStream_t st)
{
#define CALL(L) design_t<L>(a, st)
    MSOSM_DISPATCH(log2n, CALL)
#undef CALL
    return cudaErrorInvalidValue;
}

static unsigned int blocks_for(size_t n, unsigned int t) { return (unsigned int)((n + t - 1) / t); }

cudaError_t launch_fold_reduce(const float *pm, const float *pp, int D, int R, int nbins, int pend_row,
                               const int *status, double *am, double *ap, cudaStream_t st)
{
    const long long n = (long long)D * nbins;
    // from 16384 values on, 128 blocks of the 16-byte form have work enough
    if (n >= 16384 && n % 4 == 0) {
        fold_reduce4_kernel<<<blocks_for((size_t)n / 4, 32), 256, 0, st>>>(
            reinterpret_cast<const float4 *>(pm), reinterpret_cast<const float4 *>(pp), n / 4, R, pend_row, status, am,
            ap);
        return cudaGetLastError();
    }
    const unsigned int blocks = blocks_for((size_t)n, 32);
    // row groups: the largest power of two <= min(R, 32)
    if (R >= 32)
        fold_reduce_kernel<32><<<blocks, 32 * 32, 0, st>>>(pm, pp, n, R, pend_row, status, am, ap);
    else if (R >= 16)
        fold_reduce_kernel<16><<<blocks, 32 * 16, 0, st>>>(pm, pp, n, R, pend_row, status, am, ap);
    else if (R >= 8)
        fold_reduce_kernel<8><<<blocks, 32 * 8, 0, st>>>(pm, pp, n, R, pend_row, status, am, ap);
    else if (R >= 4)
        fold_reduce_kernel<4><<<blocks, 32 * 4, 0, st>>>(pm, pp, n, R, pend_row, status, am, ap);
    else if (R >= 2)
        fold_reduce_kernel<2><<<blocks, 32 * 2, 0, st>>>(pm, pp, n, R, pend_row, status, am, ap);
    else
        fold_reduce_kernel<1><<<blocks, 32, 0, st>>>(pm, pp, n, R, pend_row, status, am, ap);
    return cudaGetLastError();
}

// Reads pinned host memory directly (mapped, unified addressing), so the
// upload is ordered on the compute stream alone and never waits behind a
// large input copy on the copy engines
__global__ void span_upload_kernel(const long long *__restrict__ h, int n, int cap, long long *__restrict__ a,
                                   long long *__restrict__ b, int *__restrict__ p, int *__restrict__ dest)
{
    const int *hp = reinterpret_cast<const int *>(h + 2 * (size_t)cap);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        a[i] = h[i];
        b[i] = h[cap + i];
        p[i] = hp[i];
        dest[i] = hp[cap + i];
    }
}

// The call's spans as a launch parameter, written to the device arrays, and
// (flush) the pending period's accumulator moved to the main one.
struct SpanTable {
    int n;
    int phase0[kSpanParam], dest[kSpanParam];
    long long a[kSpanParam], b[kSpanParam];
};

__global__ void __launch_bounds__(256) fold_begin_kernel(const __grid_constant__ SpanTable t, long long *__restrict__ a,
                                                         long long *__restrict__ b, int *__restrict__ p,
                                                         int *__restrict__ dest, double *am, double *ap, size_t n)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < (size_t)t.n) {
        a[i] = t.a[i];
        b[i] = t.b[i];
        p[i] = t.phase0[i];
        dest[i] = t.dest[i];
    }
    if (i < n) {
        am[i] += ap[i];
        ap[i] = 0.0;
    }
}

// Up to kSpanParam spans travel as the launch's parameter; more are read from
// their pinned staging (which costs a bus round trip, 6 us against 2).
cudaError_t launch_fold_begin(const FoldSpan *spans, int n, long long *host, int cap, long long *a, long long *b,
                              int *phase0, int *dest, bool flush, double *acc_main, double *acc_pend, size_t nacc,
                              cudaStream_t st, int *launches)
{
    *launches = 0;
    if (n <= kSpanParam) {
        if (n == 0 && !flush)
            return cudaSuccess;
        SpanTable t;
        t.n = n;
        for (int i = 0; i < n; ++i) {
            t.a[i] = spans[i].a;
            t.b[i] = spans[i].b;
            t.phase0[i] = spans[i].phase0;
            t.dest[i] = spans[i].dest;
        }
        const size_t work = flush ? (nacc > (size_t)n ? nacc : (size_t)n) : (size_t)n;
        *launches = 1;
        fold_begin_kernel<<<blocks_for(work, 256), 256, 0, st>>>(t, a, b, phase0, dest, acc_main, acc_pend,
                                                                 flush ? nacc : 0);
        return cudaGetLastError();
    }
    int *hp = reinterpret_cast<int *>(host + 2 * (size_t)cap);
    for (int i = 0; i < n; ++i) {
        host[i] = spans[i].a;
        host[cap + i] = spans[i].b;
        hp[i] = spans[i].phase0;
        hp[cap + i] = spans[i].dest;
    }
    // a kernel reads the staging: copies on this stream would wait behind the
    // next call's input copy on the copy engine, and the dedispersion kernel
    // with them
    void *hd = nullptr;
    cudaError_t e = cudaHostGetDevicePointer(&hd, host, 0);
    if (e != cudaSuccess)
        return e;
    const unsigned int g = blocks_for((size_t)n, 256) < 64 ? blocks_for((size_t)n, 256) : 64;
    *launches = 1;
    span_upload_kernel<<<g, 256, 0, st>>>(static_cast<const long long *>(hd), n, cap, a, b, phase0, dest);
    if ((e = cudaGetLastError()) == cudaSuccess && flush) {
        *launches = 2;
        fold_flush_kernel<<<blocks_for(nacc, 256), 256, 0, st>>>(acc_main, acc_pend, nacc);
        e = cudaGetLastError();
    }
    return e;
}

cudaError_t launch_fold_readout(const double *am, size_t n, double scale, float *out, cudaStream_t st)
{
    fold_readout_kernel<<<blocks_for(n, 256), 256, 0, st>>>(am, n, scale, out);
    return cudaGetLastError();
}

cudaError_t launch_intensity(const float2 *a, const float2 *b, float *out, size_t n, cudaStream_t st)
{
    intensity_kernel<<<blocks_for(n, 256), 256, 0, st>>>(a, b, out, n);
    return cudaGetLastError();
}

// lanes per bin of the direct fold: about eight samples each, so that a warp
// reads runs of memory
static int direct_g_shift(int bpt)
{
    int g = 0;
    while (g < 5 && (8 << g) < bpt)
        ++g;
    return g;
}

static int direct_tiles(int nbins, int bpt)
{
    const int per = 256 >> direct_g_shift(bpt);
    return (nbins + per - 1) / per;
}

// Whether a call of n samples takes the second form.  A warp of the first form
// adds one bin of one span: with fewer than about 1024 of those the chunk waits
// for them.  2^22 samples, bins of 20000: 104 us a call in the first form, 54 in
// the second; 2^20 of 10937: 65 and 40; 2^22 of 3100 (1353 warps): 42 and 50.
static bool fold_wide(int bpt, int trials, long long n)
{
    return bpt > 4096 || (bpt > 1024 && n / bpt * trials < 1024);
}

int fold_direct_rows(int nbins, int bpt, int trials, int max_spans, long long n)
{
    if (fold_wide(bpt, trials, n)) {
        // rows of 4096 samples, 1200 blocks in all at most; 2^24 partial sums
        const long long R = std::min(std::min(n / 4096, 1200ll / trials), (1ll << 24) / ((long long)nbins * trials));
        return (int)std::max(R, 1ll);
    }
    const long long tiles = (long long)direct_tiles(nbins, bpt) * trials;
    const long long R = 1200 / tiles;
    return (int)(R < 1 ? 1 : (R > max_spans ? max_spans : R));
}

int fold_direct_pend_row(int bpt, int R, int trials, long long n, const FoldSpan *spans, int nspans)
{
    if (nspans == 0 || spans[nspans - 1].dest != 2)
        return R;
    int r = R - 1;  // the last share of the spans
    if (fold_wide(bpt, trials, n))  // the row the period begins in
        while (r > 0 && n * r / R > spans[nspans - 1].a)
            --r;
    return r;
}

cudaError_t launch_fold_direct(const float *I, long long n, int R, const FoldArgs &args, int trials, cudaStream_t st)
{
    FoldArgs f = args;
    if (fold_wide(f.bpt, trials, n)) {
        fold_wide_kernel<<<dim3((unsigned)R, (unsigned)trials), 256, 0, st>>>(I, n, f);
        return cudaGetLastError();
    }
    f.g_shift = direct_g_shift(f.bpt);
    fold_direct_kernel<<<dim3((unsigned)direct_tiles(f.nbins, f.bpt), (unsigned)R, (unsigned)trials), 256, 0, st>>>(I, n,
                                                                                                                   f);
    return cudaGetLastError();
}

cudaError_t launch_encode_u16(const float2 *src, uint32_t *dst, size_t n, cudaStream_t st)
{
    encode_u16_kernel<<<blocks_for(n, 256), 256, 0, st>>>(src, dst, n);
    return cudaGetLastError();
}

}  // namespace msosm

// fold_dev.cuh -- device side of the deterministic fold shared by the fused
// dedispersion kernels (CUDA-core and tensor-core) and the series fold.
#pragma once

#include "kernels.hpp"

namespace msosm {

// Folding inside the dedispersion kernel.  The host fold planner cuts each
// call's output samples into spans (one period each, sorted); a work item
// keeps a window of them in shared memory and its two partial profiles
// (complete periods, pending period) in shared memory too.  The samples of a
// step go span piece by span piece: every bin of the piece is summed by a
// group of G lanes strided over its samples, which then reduce with a fixed
// xor butterfly.  The summation order is fixed, so the result does not depend
// on scheduling.
struct FoldSmem {
    float *prof_main, *prof_pend;  // [nbins] each (or the global rows)
    int *wa, *wb, *wp, *wd;        // span window (chunk-local sample indices < 2^31)
};

// Shared-memory layout of the fold state at `base` (sized by fold_smem_bytes).
__device__ __forceinline__ void fold_smem_layout(FoldSmem &w, void *base, const FoldArgs &f)
{
    w.wa = reinterpret_cast<int *>(base);
    w.wb = w.wa + f.span_cap;
    w.wp = w.wb + f.span_cap;
    w.wd = w.wp + f.span_cap;
    w.prof_main = reinterpret_cast<float *>(w.wd + f.span_cap);
    w.prof_pend = w.prof_main + f.nbins;
}

__device__ __forceinline__ int span_lower_bound(const long long *b, int n, long long t)
{
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (b[mid] <= t)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// Load spans [at, at + cap) into the window (all threads; barriers inside).
__device__ __forceinline__ void span_refill(const FoldArgs &f, FoldSmem &w, int at, int &base, int &cnt)
{
    __syncthreads();
    const int n = min(f.span_cap, f.nspans - at);
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        w.wa[i] = (int)f.span_a[at + i];
        w.wb[i] = (int)f.span_b[at + i];
        w.wp[i] = f.span_phase0[at + i];
        w.wd[i] = f.span_dest[at + i];
    }
    base = at;
    cnt = n;
    __syncthreads();
}

// floor(x / bpt) for x >= 0 with x / bpt < 2^22 (at most nbins + 1; the host
// bounds nbins) from a float reciprocal, corrected to exact
__device__ __forceinline__ int div_bpt(int x, int bpt, float inv_bpt)
{
    if (bpt == 1)
        return x;
    int q = __float2int_rz((float)x * inv_bpt);
    if (q * bpt > x)
        --q;
    else if ((q + 1) * bpt <= x)
        ++q;
    return q;
}

// Layouts of the intensity buffer (sample t of the buffer at index ...), so
// that lanes reading bins of any length one sample at a time mostly hit
// different banks:
//  kIbufPadded: t + t/32, one pad slot per 32 samples
//  kIbufPadded2: t + 2 (t/64), which keeps even t 8-byte aligned
constexpr int kIbufPadded = 1, kIbufPadded2 = 2;
__device__ __forceinline__ int ipad(int t) { return t + (t >> 5); }
__device__ __forceinline__ int ipad2(int t) { return t + ((t >> 6) << 1); }
template <int L>
__device__ __forceinline__ int iidx(int t) { return L == kIbufPadded ? ipad(t) : ipad2(t); }

// Where a work item stands in the call's spans: span sp, held in registers,
// of a window [base, base + cnt) in shared memory.
struct FoldCursor {
    int sp, base, cnt;
    int a, b, ph, dest;  // span sp: samples [a, b), phase of a, destination (b = a = none left)
};

__device__ __forceinline__ void cursor_load(const FoldArgs &f, FoldSmem &w, FoldCursor &c)
{
    if (c.sp >= f.nspans) {
        c.a = c.b = 0x7fffffff;
        return;
    }
    if (c.sp < c.base || c.sp >= c.base + c.cnt)
        span_refill(f, w, c.sp, c.base, c.cnt);
    const int i = c.sp - c.base;
    c.a = w.wa[i];
    c.b = w.wb[i];
    c.ph = w.wp[i];
    c.dest = w.wd[i];
}

// The cursor at the first span ending after sample t (all threads).
__device__ __forceinline__ void cursor_init(const FoldArgs &f, FoldSmem &w, FoldCursor &c, long long t)
{
    c.sp = span_lower_bound(f.span_b, f.nspans, t);
    c.base = c.cnt = 0;
    span_refill(f, w, c.sp, c.base, c.cnt);
    cursor_load(f, w, c);
}

// One span piece: the sample of phase p, ph_lo <= p < ph_hi, sits at offset
// off + p.  Bin after bin goes to a group of G = 2^g_shift lanes
// (fold_g_shift), lane l taking samples l, l + G, ... in four interleaved
// sums; the group then reduces with a fixed xor butterfly.  A piece with
// fewer bins than the block has groups leaves its last warps out; `rot` (a
// multiple of 32) moves the first group to another warp with every step.
// Bound by issue: a load, an add and an address per sample.  The form before
// this one (each thread 16 consecutive samples into at most two bins, partial
// sums to shared memory, a barrier, bins completed from them) took 18
// instructions a sample, a fifth of the FP32 kernel at 4096 points.
template <int L>
__device__ __forceinline__ void fold_piece(const FoldArgs &f, float *prof, const float *ibuf, int off,
                                           int ph_lo, int ph_hi, int rot)
{
    const int G = 1 << f.g_shift;
    const int vt = ((int)threadIdx.x + rot) & ((int)blockDim.x - 1);  // blockDim a power of two
    int gw = (vt & ~31) >> f.g_shift;                                 // the warp's first group
    // at most (ph_hi - ph_lo) / bpt + 2 bins (inv_bpt may be an ulp off: + 3)
    if (gw > (int)((float)(ph_hi - ph_lo) * f.inv_bpt) + 3)
        return;
    const int l = vt & (G - 1), ngroups = (int)blockDim.x >> f.g_shift;
    const int b_lo = div_bpt(ph_lo, f.bpt, f.inv_bpt);
    int bin = b_lo + (vt >> f.g_shift), bw = b_lo + gw;
    for (; bw < f.nbins && bw * f.bpt < ph_hi; bw += ngroups, bin += ngroups) {  // whole warps
        const int s0 = bin * f.bpt;
        float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
        const bool mine = bin < f.nbins && s0 < ph_hi;
        if (mine) {
            int p = off + max(ph_lo, s0) + l;
            const int e = off + min(ph_hi, s0 + f.bpt);
            for (; p + 3 * G < e; p += 4 * G) {
                a0 += ibuf[iidx<L>(p)];
                a1 += ibuf[iidx<L>(p + G)];
                a2 += ibuf[iidx<L>(p + 2 * G)];
                a3 += ibuf[iidx<L>(p + 3 * G)];
            }
            if (p < e)
                a0 += ibuf[iidx<L>(p)];
            if (p + G < e)
                a1 += ibuf[iidx<L>(p + G)];
            if (p + 2 * G < e)
                a2 += ibuf[iidx<L>(p + 2 * G)];
        }
        float sum = (a0 + a1) + (a2 + a3);
        for (int o = G >> 1; o > 0; o >>= 1)
            sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (mine && l == 0)
            prof[bin] += sum;
    }
}

// Fold the n intensities of a step (ibuf: chunk-local samples t0..t0+n-1);
// the cursor stands at or before the first span ending after t0.
template <int L>
__device__ __forceinline__ void fold_block(const FoldArgs &f, FoldSmem &w, const float *ibuf, int t0, int n,
                                           FoldCursor &c, int rot = 0)
{
    const int t1 = t0 + n;
    while (c.b <= t0) {
        ++c.sp;
        cursor_load(f, w, c);
    }
    while (c.a < t1) {
        const int a = max(c.a, t0), b = min(c.b, t1);
        if (c.dest != 0 && a < b) {
            const int ph_lo = c.ph + (a - c.a);
            fold_piece<L>(f, c.dest == 1 ? w.prof_main : w.prof_pend, ibuf, a - t0 - ph_lo, ph_lo, ph_lo + (b - a),
                          rot);
        }
        if (c.b >= t1)
            break;
        // a later span of this step may fold into the same bins
        __syncthreads();
        ++c.sp;
        cursor_load(f, w, c);
    }
}

}  // namespace msosm

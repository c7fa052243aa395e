// Sliding-window moments of a source's coverage on one chromosome (K4-K7): build_depth_signal
// (src/fourier/depth.rs:109-215) and moments_from_signal (src/fourier/moments.rs:192-466).
//
// K4  depth signal g[0..N) in f32, bit for bit the reference's: the fractional-bin impulses are
//     summed per bin in the reference's order (all start spikes, then all end spikes, each in input
//     order) and the prefix sum follows simd_cumsum_f32's chunk-of-8 order, including its
//     sequential f32 carry chain (only chunks with a non-zero total change the carry, so the chain
//     runs over the compacted non-zero totals).  The f32 rounding residues of g move large-window
//     means by ~1e-4 relative, so any other summation order could not match the reference.
// K5  centred signal u = g - mean(g) and its prefix sum U (tile sums, one block over them, a scan in each
//     tile; sums in double-double, or float-float).
// K6  autocorrelation A[m] = sum_k u[k] u[k+m] by a hand-written Stockham FFT (passes of radix 16 to 256
//     through shared memory): FFT(u zero-padded to M = 2^ceil(log2 2N)), |X|^2, FFT again, real part / M, each as a
//     complex transform of M / 2 packed points.
// K7  window moments for the L grid of the compact store:
//       sum_j F_L(j)   = (UU(N+1) - UU(L)) - UU(N-L+1)                    (UU = prefix of U)
//       sum_j F_L(j)^2 = L A[0] + 2 (L P0(L) - P1(L)) - Q(L-1) - V(L-1)
//     with F_L(j) the window sums of u, P0/P1 prefix sums of A[m] and m A[m] (m >= 1), Q the prefix
//     sum of U[t]^2 and V that of (U[N] - U[N-t])^2 (the partial windows at both ends of the full
//     linear convolution).  mean(L) = L mean(g) + sum F / n_w, var(L) = sum F^2 / n_w - (sum F /
//     n_w)^2 in FP64, clamped at 0 as the reference does.  Every term is bounded by the centred
//     signal, so the cancellation that the reference's d*-autocorrelation suffers (~1e10,
//     docs/todo.md) does not arise.  The prefix sums are taken at the grid's points only, from sums over
//     tiles: in double-double over the tiles and for U, in the tiles in double-double, or in float-float for
//     the other terms of the compensated path.
#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "internal.h"

namespace rgl {

std::vector<uint64_t> moment_grid(uint64_t n);

struct DD {
    double hi, lo;
};
__host__ __device__ __forceinline__ DD dd_two_sum(double a, double b) {
    const double s = a + b;
    const double bb = s - a;
    const double e = (a - (s - bb)) + (b - bb);
    return DD{s, e};
}
__host__ __device__ __forceinline__ DD dd_add(DD a, DD b) {
    DD s = dd_two_sum(a.hi, b.hi);
    const DD t = dd_two_sum(a.lo, b.lo);
    s.lo += t.hi;
    s = dd_two_sum(s.hi, s.lo);
    s.lo += t.lo;
    return dd_two_sum(s.hi, s.lo);
}
__device__ __forceinline__ DD dd_neg(DD a) { return DD{-a.hi, -a.lo}; }
__device__ __forceinline__ DD dd_mul_d(DD a, double b) {
    const double p = a.hi * b;
    double e = fma(a.hi, b, -p);
    e = fma(a.lo, b, e);
    return dd_two_sum(p, e);
}

// ---- K4: impulses ---------------------------------------------------------------------------------
// Two records per interval end: (bin, impulse), or (n_bins, 0) where there is none.  The start records
// of all intervals come first, in input order, then the end records, and an interval's two records of
// one phase never share a bin: a stable sort by bin alone leaves every bin's records in the
// reference's order.  32-bit keys over the bits of n_bins take 3 radix passes (chr1 at 100 bp); the
// order spelled out in 64-bit keys took 8 (1.6e6 records: 171 us, now 65).
__global__ void k_spike_records(uint32_t n, const rgl_interval* __restrict__ iv, uint32_t n_bins, uint32_t bin,
                                uint32_t* __restrict__ key, float* __restrict__ val) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t max_bp = n_bins * bin;  // build_spikes clip (src/fourier/depth.rs:206-215), u32 arithmetic
#pragma unroll
    for (uint32_t phase = 0; phase < 2; phase++) {
        const uint32_t x0 = phase ? iv[i].end : iv[i].start;
        const uint32_t x = x0 < max_bp ? x0 : max_bp;
        const uint32_t b = x / bin;
        const float frac = __fdiv_rn((float)(x % bin), (float)bin);
        const float c1 = __fsub_rn(1.0f, frac);
        const uint64_t j = 2ull * ((uint64_t)phase * n + i);  // key and val are 8-byte aligned there
        const bool a = b < n_bins, c = frac > 0.0f && b + 1 < n_bins;
        *reinterpret_cast<uint2*>(key + j) = make_uint2(a ? b : n_bins, c ? b + 1 : n_bins);
        *reinterpret_cast<float2*>(val + j) =
            make_float2(a ? (phase ? -c1 : c1) : 0.f, c ? (phase ? -frac : frac) : 0.f);
    }
}

// Bits of the records' keys: 0 .. n_bins.
static int spike_key_bits(uint64_t n_bins) {
    int bits = 1;
    while (bits < 32 && (1ull << bits) <= n_bins) bits++;
    return bits;
}

// One thread per run of equal bins in the sorted records: the bin's impulse, summed in f32 in the
// reference's order.
__global__ void k_bin_sums(uint64_t m, uint32_t n_bins, const uint32_t* __restrict__ key,
                           const float* __restrict__ val, float* __restrict__ g) {
    const uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (j >= m) return;
    const uint32_t b = key[j];
    if (b >= n_bins || (j > 0 && key[j - 1] == b)) return;
    float s = 0.0f;
    for (uint64_t k = j; k < m && key[k] == b; k++) s = __fadd_rn(s, val[k]);
    g[b] = s;
}

// ---- K4: simd_cumsum_f32 (src/fourier/depth.rs:143-204) in its own order ------------------------------
__global__ void k_chunk_local(uint64_t full, float* __restrict__ g, float* __restrict__ totals,
                              uint8_t* __restrict__ nz) {
    const uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (c >= full) return;
    float v[8];
    const float4* p = reinterpret_cast<const float4*>(g + 8 * c);
    const float4 a = p[0], b = p[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
#pragma unroll
    for (int i = 1; i < 8; i++) v[i] = __fadd_rn(v[i], v[i - 1]);
    float4* q = reinterpret_cast<float4*>(g + 8 * c);
    q[0] = make_float4(v[0], v[1], v[2], v[3]);
    q[1] = make_float4(v[4], v[5], v[6], v[7]);
    totals[c] = v[7];
    nz[c] = v[7] != 0.0f;
}

// The sequential f32 carry over the chunks whose total is non-zero (adding an exact zero leaves
// the carry unchanged), then the tail elements, exactly as the reference orders them.
// Bound: the dependent f32 additions, about four clocks each (no other order gives the reference's
// roundings).  One lane adds from shared memory, four totals per read, while the other warps gather
// the next stage and store the one before, so that the chain never waits for memory.  One thread
// reading idx and totals from global memory took 8.66 ms for 3.1e5 chunks (4e5 intervals on 2.5e6
// bins), 0.14 ms for 8e3; staged so 0.63 ms (four clocks each) and 0.02 ms.
constexpr int kChainStage = 2048, kChainThreads = 512;
__global__ void __launch_bounds__(kChainThreads) k_carry_chain(const int* __restrict__ count,
                                                               const uint32_t* __restrict__ idx,
                                                               const float* __restrict__ totals,
                                                               float* __restrict__ cum_after, float* __restrict__ g,
                                                               uint64_t n, uint64_t full) {
    __shared__ __align__(16) float in[2][kChainStage];
    __shared__ __align__(16) float out[2][kChainStage];
    const int cnt = *count, stages = (cnt + kChainStage - 1) / kChainStage;
    auto load = [&](int s, int first, int step) {  // zeros past the last total leave the carry as it is
        for (int i = first; i < kChainStage; i += step) {
            const int k = s * kChainStage + i;
            in[s & 1][i] = k < cnt ? totals[idx[k]] : 0.0f;
        }
    };
    auto store = [&](int s, int first, int step) {
        for (int i = first; i < kChainStage; i += step) {
            const int k = s * kChainStage + i;
            if (k < cnt) cum_after[k] = out[s & 1][i];
        }
    };
    if (stages) load(0, threadIdx.x, kChainThreads);
    __syncthreads();
    float carry = 0.0f;  // thread 0's
    for (int s = 0; s < stages; s++) {
        if (threadIdx.x == 0) {
            const float4* v = reinterpret_cast<const float4*>(in[s & 1]);
            float4* o = reinterpret_cast<float4*>(out[s & 1]);
            // sixteen totals a step, the next sixteen read before the additions of this step begin
            const int steps = (min(cnt - s * kChainStage, kChainStage) + 15) / 16;
            float4 cur[4];
#pragma unroll
            for (int h = 0; h < 4; h++) cur[h] = v[h];
            for (int q = 0; q < steps; q++) {
                const float4* w = v + 4 * min(q + 1, kChainStage / 16 - 1);
                float4 next[4];
#pragma unroll
                for (int h = 0; h < 4; h++) next[h] = w[h];
#pragma unroll
                for (int h = 0; h < 4; h++) {
                    float4 a = cur[h];
                    a.x = carry = __fadd_rn(carry, a.x);
                    a.y = carry = __fadd_rn(carry, a.y);
                    a.z = carry = __fadd_rn(carry, a.z);
                    a.w = carry = __fadd_rn(carry, a.w);
                    o[4 * q + h] = a;
                    cur[h] = next[h];
                }
            }
        } else if (threadIdx.x >= 32) {
            if (s + 1 < stages) load(s + 1, threadIdx.x - 32, kChainThreads - 32);
            if (s > 0) store(s - 1, threadIdx.x - 32, kChainThreads - 32);
        }
        __syncthreads();
    }
    if (stages) store(stages - 1, threadIdx.x, kChainThreads);
    if (threadIdx.x == 0) {
        const uint64_t tail = full * 8;
        for (uint64_t i = tail + 1; i < n; i++) g[i] = __fadd_rn(g[i], g[i - 1]);
        if (full > 0 && tail < n && carry != 0.0f)
            for (uint64_t i = tail; i < n; i++) g[i] = __fadd_rn(g[i], carry);
    }
}

// One thread per chunk: one search serves its eight bins (one per bin: 33 us for 2.5e6 bins; now 10).
__global__ void k_apply_carry(uint64_t full, const int* __restrict__ count, const uint32_t* __restrict__ idx,
                              const float* __restrict__ cum_after, float* __restrict__ g) {
    const uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (c >= full || c == 0) return;  // the reference adds no carry to chunk 0
    // carries[c] = running sum of the totals of chunks < c = cum_after of the last non-zero chunk < c
    int lo = 0, hi = *count;  // number of compacted chunks with index < c
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (idx[mid] < c) lo = mid + 1; else hi = mid;
    }
    const float carry = lo ? cum_after[lo - 1] : 0.0f;
    float4* p = reinterpret_cast<float4*>(g + 8 * c);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        float4 a = p[h];
        a.x = __fadd_rn(a.x, carry);
        a.y = __fadd_rn(a.y, carry);
        a.z = __fadd_rn(a.z, carry);
        a.w = __fadd_rn(a.w, carry);
        p[h] = a;
    }
}

__device__ __forceinline__ DD dd_mul(DD a, DD b) {
    const double p = a.hi * b.hi;
    double e = fma(a.hi, b.hi, -p);
    e = fma(a.hi, b.lo, e);
    e = fma(a.lo, b.hi, e);
    return dd_two_sum(p, e);
}
__device__ __forceinline__ DD dd_div_d(DD a, double b) {
    const double q = a.hi / b;
    const DD r = dd_add(a, dd_neg(dd_mul_d(DD{q, 0.0}, b)));
    return dd_two_sum(q, (r.hi + r.lo) / b);
}
template <typename UT>
__device__ __forceinline__ DD u_at(const UT* U, uint64_t i);
template <>
__device__ __forceinline__ DD u_at<double>(const double* U, uint64_t i) { return DD{U[i], 0.0}; }

// ---- the compensated-FP32 path (K5-K7 with float-float arithmetic) ------------------------------
// Every value is an unevaluated sum hi + lo of two floats (|lo| <= ulp(hi) / 2), about 48 bits of
// significand, kept by the error-free transformations two-sum (Knuth) and two-product (one FMA)
// as in Dekker's double-length arithmetic (T. J. Dekker, "A floating-point technique for extending
// the available precision", Numer. Math. 18, 1971; Y. Hida, X. S. Li, D. H. Bailey, "Algorithms for
// quad-double precision floating point arithmetic", ARITH 2001, for the add / mul sequences).  The
// centred signal is scaled by a power of two per chromosome so that it is O(1) (no denormal lo
// parts), and the FFT, the power spectrum and the sums inside a tile run in float-float.  FP64 appears in
// the twiddles (sincospi, split into two floats), in the sums over the tiles and of U (double-double), and
// when the per-L results are combined (k_window_moments: the final reduction and the variance subtraction).
struct __align__(8) FF {
    float hi, lo;
};
struct __align__(16) CFF {
    FF re, im;
};
__device__ __forceinline__ FF ff_two_sum(float a, float b) {
    const float s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
    return FF{s, e};
}
__device__ __forceinline__ FF ff_quick(float a, float b) {  // |a| >= |b|
    const float s = __fadd_rn(a, b);
    return FF{s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ FF ff_add(FF a, FF b) {
    FF s = ff_two_sum(a.hi, b.hi);
    const FF t = ff_two_sum(a.lo, b.lo);
    s.lo = __fadd_rn(s.lo, t.hi);
    s = ff_quick(s.hi, s.lo);
    s.lo = __fadd_rn(s.lo, t.lo);
    return ff_quick(s.hi, s.lo);
}
__device__ __forceinline__ FF ff_neg(FF a) { return FF{-a.hi, -a.lo}; }
__device__ __forceinline__ FF ff_sub(FF a, FF b) { return ff_add(a, ff_neg(b)); }
__device__ __forceinline__ FF ff_mul(FF a, FF b) {
    const float p = __fmul_rn(a.hi, b.hi);
    float e = __fmaf_rn(a.hi, b.hi, -p);
    e = __fmaf_rn(a.hi, b.lo, e);
    e = __fmaf_rn(a.lo, b.hi, e);
    return ff_quick(p, e);
}
__device__ __forceinline__ FF ff_from_double_exact(uint64_t t) {  // an integer below 2^48, exactly
    const float hi = (float)(t & ~0xFFFFFFull);                    // the top bits (exact in a float)
    return ff_two_sum(hi, (float)(t & 0xFFFFFFull));
}
__device__ __forceinline__ CFF cff_add(CFF a, CFF b) { return CFF{ff_add(a.re, b.re), ff_add(a.im, b.im)}; }
__device__ __forceinline__ CFF cff_sub(CFF a, CFF b) { return CFF{ff_sub(a.re, b.re), ff_sub(a.im, b.im)}; }
__device__ __forceinline__ CFF cff_mul(CFF a, CFF b) {
    return CFF{ff_sub(ff_mul(a.re, b.re), ff_mul(a.im, b.im)), ff_add(ff_mul(a.re, b.im), ff_mul(a.im, b.re))};
}
template <>
__device__ __forceinline__ DD u_at<FF>(const FF* U, uint64_t i) {
    return dd_two_sum((double)U[i].hi, (double)U[i].lo);
}

// ---- K5, K7: prefix sums at the grid's points ------------------------------------------------------
// The window moments need prefix sums of five terms (A[t], t A[t], U[t]^2, (U[N] - U[N-t])^2, U[t]) at
// the grid's ~1,000 points only, so no prefix is written out: one pass sums tiles of the terms, one
// block per term scans the tile sums, and one block per grid point adds the part of its last tile.
// Bound: one read of A and U (16 to 24 bytes a bin), from L2 at these sizes.  Five device-wide scans of
// 16-byte pairs, each over an array of terms written first, took 580 us at 2.5e6 bins (FP64); the
// three kernels take 86.
//
// Both arithmetics run the same kernels: P64 sums doubles in double-double, PFF sums float-float
// values in float-float.
struct P64 {
    using S = double;   // a value of the signal
    using C = double2;  // a complex value
    using T = DD;       // a sum
    static __device__ __forceinline__ S re(C a) { return a.x; }
    static __device__ __forceinline__ S im(C a) { return a.y; }
    static __device__ __forceinline__ C pack(S re, S im) { return make_double2(re, im); }
    static __device__ __forceinline__ C conj(C a) { return make_double2(a.x, -a.y); }
    static __device__ __forceinline__ C half(C a) { return make_double2(0.5 * a.x, 0.5 * a.y); }
    static __device__ __forceinline__ S norm(C a) { return a.x * a.x + a.y * a.y; }
    static __device__ __forceinline__ S addv(S a, S b) { return a + b; }
    static __device__ __forceinline__ S scaled(S a, uint64_t m) { return a * (1.0 / (double)m); }  // m a power of two
    static __device__ __forceinline__ T zero() { return DD{0.0, 0.0}; }
    static __device__ __forceinline__ T add(T a, T b) { return dd_add(a, b); }
    static __device__ __forceinline__ T add_s(T a, S v) {
        const DD s = dd_two_sum(a.hi, v);
        return dd_two_sum(s.hi, s.lo + a.lo);
    }
    static __device__ __forceinline__ S sub(S a, S b) { return a - b; }
    static __device__ __forceinline__ S mul(S a, S b) { return a * b; }
    static __device__ __forceinline__ S of_index(uint64_t t) { return (double)t; }
    static __device__ __forceinline__ S none() { return 0.0; }
    static __device__ __forceinline__ DD sum_dd(T a, int) { return a; }
    static __device__ __forceinline__ double value(S a, int) { return a; }
};
struct PFF {
    using S = FF;
    using C = CFF;
    using T = FF;
    static __device__ __forceinline__ S re(C a) { return a.re; }
    static __device__ __forceinline__ S im(C a) { return a.im; }
    static __device__ __forceinline__ C pack(S re, S im) { return CFF{re, im}; }
    static __device__ __forceinline__ C conj(C a) { return CFF{a.re, ff_neg(a.im)}; }
    static __device__ __forceinline__ C half(C a) {
        return CFF{FF{0.5f * a.re.hi, 0.5f * a.re.lo}, FF{0.5f * a.im.hi, 0.5f * a.im.lo}};
    }
    static __device__ __forceinline__ S norm(C a) { return ff_add(ff_mul(a.re, a.re), ff_mul(a.im, a.im)); }
    static __device__ __forceinline__ S addv(S a, S b) { return ff_add(a, b); }
    static __device__ __forceinline__ S scaled(S a, uint64_t m) {
        const float r = 1.0f / (float)m;  // exact
        return FF{a.hi * r, a.lo * r};
    }
    static __device__ __forceinline__ T zero() { return FF{0.f, 0.f}; }
    static __device__ __forceinline__ T add(T a, T b) { return ff_add(a, b); }
    static __device__ __forceinline__ T add_s(T a, S v) { return ff_add(a, v); }
    static __device__ __forceinline__ S sub(S a, S b) { return ff_sub(a, b); }
    static __device__ __forceinline__ S mul(S a, S b) { return ff_mul(a, b); }
    static __device__ __forceinline__ S of_index(uint64_t t) { return ff_from_double_exact(t); }
    static __device__ __forceinline__ S none() { return FF{0.f, 0.f}; }
    // a sum in double-double, scaled back by the exact power of two 2^sc
    static __device__ __forceinline__ DD sum_dd(T a, int sc) {
        return DD{ldexp((double)a.hi, sc), ldexp((double)a.lo, sc)};
    }
    static __device__ __forceinline__ double value(S a, int sc) { return ldexp((double)a.hi + (double)a.lo, sc); }
};
template <class P>
struct SumOp {
    __device__ __forceinline__ typename P::T operator()(const typename P::T& a, const typename P::T& b) const {
        return P::add(a, b);
    }
};

template <class P>
__device__ __forceinline__ typename P::T warp_sum(typename P::T v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        typename P::T w;
        w.hi = __shfl_down_sync(0xffffffffu, v.hi, o);
        w.lo = __shfl_down_sync(0xffffffffu, v.lo, o);
        v = P::add(v, w);
    }
    return v;  // lane 0's
}

// ---- K6: the autocorrelation by two real transforms -------------------------------------------------
// The signal is real and its power spectrum real and even, so both transforms of length M run as complex
// transforms of H = M / 2 points over packed pairs (even elements real parts, odd elements imaginary),
// untangled afterwards: X[k] = E + W^k O, X[H-k] = conj(E - W^k O), E = (Z[k] + conj Z[H-k]) / 2,
// O = (Z[k] - conj Z[H-k]) / 2i, W = exp(-2 pi i / M).
//
// One pass is a step of the out-of-place Stockham formulation (Govindaraju et al., "High performance
// discrete Fourier transforms on graphics processors", SC 2008) with radix R = 16 R2 <= 256: column j
// gathers R elements at stride H/R, twiddles them by exp(-2 pi i (j mod Ns) r / (Ns R)), transforms them
// and scatters to (j / Ns) Ns R + (j mod Ns) + k Ns.  A block takes 256 / R2 neighbouring columns: each
// thread does a 16-point transform in registers, the block exchanges through shared memory, and the
// R2-point transforms finish the column, so that reads and writes of neighbouring columns coalesce and
// 2^22 points take three passes over memory instead of six (one 16-point transform a pass) and half the
// points.  Bound: FP64 by HBM / L2 traffic (32 bytes a point a pass), float-float by FP32 issue.
// Both transforms with the spectrum and the autocorrelation: FP64 at 2.5e6 bins (M = 2^23) 720 -> 250 us,
// float-float at 2.1e6 bins (M = 2^22) 1,150 -> 375 us.
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cmul(double2 a, double2 w) {
    return make_double2(a.x * w.x - a.y * w.y, a.x * w.y + a.y * w.x);
}
__device__ __forceinline__ double2 crot(double2 a) { return make_double2(a.y, -a.x); }  // times -i
__device__ __forceinline__ CFF cadd(CFF a, CFF b) { return cff_add(a, b); }
__device__ __forceinline__ CFF csub(CFF a, CFF b) { return cff_sub(a, b); }
__device__ __forceinline__ CFF cmul(CFF a, CFF w) { return cff_mul(a, w); }
__device__ __forceinline__ CFF crot(CFF a) { return CFF{a.im, ff_neg(a.re)}; }
// times exp(-i pi / 4) and exp(-3 i pi / 4)
constexpr double kHalfRoot = 0.70710678118654752440;
__device__ __forceinline__ double2 crot45(double2 a) {
    return make_double2(kHalfRoot * (a.x + a.y), kHalfRoot * (a.y - a.x));
}
__device__ __forceinline__ double2 crot135(double2 a) {
    return make_double2(kHalfRoot * (a.y - a.x), -kHalfRoot * (a.x + a.y));
}
__device__ __forceinline__ FF ff_const(double v) { return FF{(float)v, (float)(v - (double)(float)v)}; }
__device__ __forceinline__ CFF crot45(CFF a) {
    const FF h = ff_const(kHalfRoot);
    return CFF{ff_mul(h, ff_add(a.re, a.im)), ff_mul(h, ff_sub(a.im, a.re))};
}
__device__ __forceinline__ CFF crot135(CFF a) {
    const FF h = ff_const(kHalfRoot);
    return CFF{ff_mul(h, ff_sub(a.im, a.re)), ff_neg(ff_mul(h, ff_add(a.re, a.im)))};
}
__device__ __forceinline__ void cset(double2& w, double c, double s) { w = make_double2(c, s); }
__device__ __forceinline__ void cset(CFF& w, double c, double s) { w = CFF{ff_const(c), ff_const(s)}; }

// b times exp(-2 pi i K / 16), K < 8.
template <int K, class C>
__device__ __forceinline__ C ctw16(C b) {
    constexpr double c1 = 0.92387953251128675613, s1 = 0.38268343236508977173;  // cos, sin of pi / 8
    if constexpr (K == 0) return b;
    else if constexpr (K == 4) return crot(b);
    else if constexpr (K == 2) return crot45(b);
    else if constexpr (K == 6) return crot135(b);
    else {
        C w;
        cset(w, K == 1 ? c1 : K == 3 ? s1 : K == 5 ? -s1 : -c1, (K == 1 || K == 7) ? -s1 : -c1);
        return cmul(b, w);
    }
}
template <int LEN, int K, int R, class C>
__device__ __forceinline__ void dft_level(C* v) {
    if constexpr (K < LEN / 2) {
#pragma unroll
        for (int i = 0; i < R; i += LEN) {
            const C a = v[i + K], t = ctw16<K*(16 / LEN)>(v[i + K + LEN / 2]);
            v[i + K] = cadd(a, t);
            v[i + K + LEN / 2] = csub(a, t);
        }
        dft_level<LEN, K + 1, R>(v);
    }
}
template <int LEN, int R, class C>
__device__ __forceinline__ void dft_levels(C* v) {
    if constexpr (LEN <= R) {
        dft_level<LEN, 0, R>(v);
        dft_levels<2 * LEN, R>(v);
    }
}
// In-register transform of R <= 16 points (radix-2 decimation in time), natural order in and out.
template <int R, class C>
__device__ __forceinline__ void dft_regs(C* v) {
#pragma unroll
    for (int i = 0; i < R; i++) {
        int j = 0;
#pragma unroll
        for (int b = 1; b < R; b <<= 1) j = (j << 1) | ((i / b) & 1);
        if (i < j) {
            const C t = v[i];
            v[i] = v[j];
            v[j] = t;
        }
    }
    dft_levels<2, R>(v);
}

// exp(-2 pi i k / 256), host-computed.
__constant__ double2 c_tw256[256];
__constant__ CFF c_tw256f[256];

// exp(-2 pi i t / M), by sincospi of the exact quotient.  The float-float path splits it in two floats
// each (2^-49): the FP64 units stand idle there, and products of coarse and fine float-float table
// entries cost two gathers and a complex float-float product more (114 us a pass of 2^21 points).
template <class P>
__device__ __forceinline__ typename P::C twiddle(uint64_t t, uint64_t M) {
    double s, c;
    sincospi(-2.0 * (double)t / (double)M, &s, &c);
    if constexpr (std::is_same<P, P64>::value) return make_double2(c, s);
    else return CFF{ff_const(c), ff_const(s)};
}
template <class P, int N>
__device__ __forceinline__ typename P::C tw_inner(int k) {  // exp(-2 pi i k / N), N <= 256
    if constexpr (std::is_same<P, P64>::value) return c_tw256[k * (256 / N)];
    else return c_tw256f[k * (256 / N)];
}

// Element idx of the packed input: 0 a complex array, 1 a real signal of n elements (zero past them), 2
// the power spectrum P[0 .. H], mirrored (P[M - k] = P[k]).
template <class P, int SRC>
__device__ __forceinline__ typename P::C fft_input(const void* __restrict__ in, uint64_t idx, uint64_t H, uint64_t n) {
    using C = typename P::C;
    using S = typename P::S;
    if constexpr (SRC == 0) return reinterpret_cast<const C*>(in)[idx];
    else {
        const S* x = reinterpret_cast<const S*>(in);
        const uint64_t i = 2 * idx;
        if constexpr (SRC == 1) {
            if (i + 1 < n) return *reinterpret_cast<const C*>(x + i);
            return P::pack(i < n ? x[i] : P::none(), P::none());
        } else {
            if (i < H) return *reinterpret_cast<const C*>(x + i);  // H is even: i + 1 < H
            return P::pack(x[2 * H - i], x[2 * H - i - 1]);
        }
    }
}

template <class P, int R2, int SRC>
__global__ void __launch_bounds__(256) k_fft_pass(const void* __restrict__ in, typename P::C* __restrict__ out,
                                                  uint64_t H, uint64_t Ns, uint64_t n) {
    using C = typename P::C;
    constexpr int R = 16 * R2, kCols = 256 / R2;
    extern __shared__ __align__(16) unsigned char fft_smem[];
    C* sm = reinterpret_cast<C*>(fft_smem);
    const uint64_t stride = H / R, j0 = blockIdx.x * (uint64_t)kCols;
    {
        const int c = threadIdx.x % kCols, b = threadIdx.x / kCols;
        const uint64_t j = j0 + c;
        C v[16];
        if (j < stride) {
#pragma unroll
            for (int a = 0; a < 16; a++) v[a] = fft_input<P, SRC>(in, j + (uint64_t)(b + R2 * a) * stride, H, n);
            if constexpr (SRC == 0) {
                const uint64_t k = j & (Ns - 1);
#pragma unroll
                for (int a = 0; a < 16; a++)
                    v[a] = cmul(v[a], twiddle<P>(k * (uint64_t)(b + R2 * a), Ns * R));
            }
        } else {
#pragma unroll
            for (int a = 0; a < 16; a++) v[a] = P::pack(P::none(), P::none());
        }
        dft_regs<16>(v);
#pragma unroll
        for (int a = 0; a < 16; a++) sm[(b * 16 + a) * kCols + c] = (a && R2 > 1) ? cmul(v[a], tw_inner<P, R>(b * a)) : v[a];
    }
    __syncthreads();
    C y[16];
#pragma unroll
    for (int e = 0; e < 16 / R2; e++) {
        const int d = threadIdx.x + 256 * e, a = d / kCols, c = d % kCols;
#pragma unroll
        for (int b = 0; b < R2; b++) y[e * R2 + b] = sm[(b * 16 + a) * kCols + c];
        dft_regs<R2>(y + e * R2);
    }
    if constexpr (SRC == 0) {
#pragma unroll
        for (int e = 0; e < 16 / R2; e++) {
            const int d = threadIdx.x + 256 * e, a = d / kCols, c = d % kCols;
            const uint64_t j = j0 + c;
            if (j < stride) {
                const uint64_t k = j & (Ns - 1);
                C* o = out + (j - k) * R + k;
#pragma unroll
                for (int b = 0; b < R2; b++) o[(uint64_t)(a + 16 * b) * Ns] = y[e * R2 + b];
            }
        }
    } else {
        // first pass (Ns = 1): a column's outputs are consecutive; stored through shared memory, column
        // by column (one element of padding each)
        __syncthreads();
#pragma unroll
        for (int e = 0; e < 16 / R2; e++) {
            const int d = threadIdx.x + 256 * e, a = d / kCols, c = d % kCols;
#pragma unroll
            for (int b = 0; b < R2; b++) sm[c * (R + 1) + a + 16 * b] = y[e * R2 + b];
        }
        __syncthreads();
        for (int x = threadIdx.x; x < kCols * R; x += 256) {
            const int c = x / R, k = x % R;
            if (j0 + c < stride) out[j0 * R + x] = sm[c * (R + 1) + k];
        }
    }
}

// Transforms of at most 16 points: one thread.
template <class P, int R, int SRC>
__global__ void k_fft_small(const void* __restrict__ in, typename P::C* __restrict__ out, uint64_t n) {
    typename P::C v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = fft_input<P, SRC>(in, r, R, n);
    dft_regs<R>(v);
#pragma unroll
    for (int r = 0; r < R; r++) out[r] = v[r];
}

// E and T = W^k O of the pair (k, H - k), 0 < k <= H / 2.
template <class P>
__device__ __forceinline__ void untangle(const typename P::C* __restrict__ Z, uint64_t k, uint64_t H,
                                         typename P::C& E, typename P::C& T) {
    using C = typename P::C;
    const C a = Z[k], b = P::conj(Z[H - k]);
    E = P::half(cadd(a, b));
    T = cmul(crot(P::half(csub(a, b))), twiddle<P>(k, 2 * H));  // D / 2i = -i D / 2
}

// The power spectrum P[0 .. H] of the packed transform Z.
template <class P>
__global__ void k_power(uint64_t H, const typename P::C* __restrict__ Z, typename P::S* __restrict__ pw) {
    const uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (k > H / 2) return;
    if (k == 0) {
        const typename P::S s = P::addv(P::re(Z[0]), P::im(Z[0])), d = P::sub(P::re(Z[0]), P::im(Z[0]));
        pw[0] = P::mul(s, s);
        pw[H] = P::mul(d, d);
        return;
    }
    typename P::C E, T;
    untangle<P>(Z, k, H, E, T);
    pw[k] = P::norm(cadd(E, T));
    pw[H - k] = P::norm(csub(E, T));
}

// A[m] = Re FFT(P)[m] / M for m < n, from the packed transform Q of the spectrum.
template <class P>
__global__ void k_autocorr(uint64_t H, uint64_t n, const typename P::C* __restrict__ Q, typename P::S* __restrict__ A) {
    const uint64_t m = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (m > H / 2) return;
    if (m == 0) {
        A[0] = P::scaled(P::addv(P::re(Q[0]), P::im(Q[0])), 2 * H);
        return;
    }
    typename P::C E, T;
    untangle<P>(Q, m, H, E, T);
    if (m < n) A[m] = P::scaled(P::addv(P::re(E), P::re(T)), 2 * H);
    if (H - m < n) A[H - m] = P::scaled(P::sub(P::re(E), P::re(T)), 2 * H);
}

// What the passes over one signal share, on the device.
struct MomentState {
    DD gsum;       // sum of g
    double gbar;   // its mean as the centring uses it (P64)
    FF gbar_ff;    // and in float-float (PFF)
    float scale;   // 2^-e (PFF): u is scaled to O(1)
    int e;
};

constexpr int kSigThreads = 256, kSigItems = 8, kSigTile = kSigThreads * kSigItems;

// Tile sums of g (and the tile's largest value, for PFF's scale).
template <class P>
__global__ void __launch_bounds__(kSigThreads) k_g_tiles(uint64_t n, const float* __restrict__ g,
                                                         typename P::T* __restrict__ tsum, float* __restrict__ tmax) {
    __shared__ typename P::T part[kSigThreads / 32];
    __shared__ float top[kSigThreads / 32];
    const uint64_t base = blockIdx.x * (uint64_t)kSigTile + threadIdx.x;
    typename P::T s = P::zero();
    float m = 0.f;
#pragma unroll
    for (int k = 0; k < kSigItems; k++) {
        const uint64_t i = base + (uint64_t)k * kSigThreads;
        const float v = i < n ? g[i] : 0.f;
        if constexpr (std::is_same<P, P64>::value) s = P::add_s(s, (double)v);
        else s = P::add_s(s, FF{v, 0.f});
        m = fmaxf(m, v);
    }
    s = warp_sum<P>(s);
#pragma unroll
    for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) {
        part[threadIdx.x >> 5] = s;
        top[threadIdx.x >> 5] = m;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kSigThreads / 32; w++) {
            s = P::add(s, part[w]);
            m = fmaxf(m, top[w]);
        }
        tsum[blockIdx.x] = s;
        tmax[blockIdx.x] = m;
    }
}

// One block: sums[0..nt) becomes its exclusive prefix sums, *total the whole.
template <class P>
__device__ __forceinline__ void scan_tiles(uint64_t nt, typename P::T* __restrict__ sums, typename P::T* total) {
    using T = typename P::T;
    using BS = cub::BlockScan<T, 1024>;
    __shared__ typename BS::TempStorage tmp;
    T run = P::zero();
    for (uint64_t b0 = 0; b0 < nt; b0 += 1024) {
        const uint64_t b = b0 + threadIdx.x;
        const T v = b < nt ? sums[b] : P::zero();
        T ex, agg;
        BS(tmp).ExclusiveScan(v, ex, P::zero(), SumOp<P>(), agg);
        if (b < nt) sums[b] = P::add(run, ex);
        run = P::add(run, agg);
        __syncthreads();
    }
    *total = run;
}

// The sum and mean of g and, for PFF, the scale: 2^e >= max(g) >= |u| (coverage is non-negative).
template <class P>
__global__ void __launch_bounds__(1024) k_g_tops(uint64_t n, uint64_t nt, typename P::T* __restrict__ tsum,
                                                 const float* __restrict__ tmax, MomentState* __restrict__ ms) {
    typename P::T total;
    scan_tiles<P>(nt, tsum, &total);
    __shared__ float top[1024];
    float m = 0.f;
    for (uint64_t b = threadIdx.x; b < nt; b += 1024) m = fmaxf(m, tmax[b]);
    top[threadIdx.x] = m;
    __syncthreads();
    for (int k = 512; k; k >>= 1) {
        if (threadIdx.x < k) top[threadIdx.x] = fmaxf(top[threadIdx.x], top[threadIdx.x + k]);
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        if constexpr (std::is_same<P, P64>::value) {
            ms->gsum = total;
            ms->gbar = total.hi / (double)n + total.lo / (double)n;
            ms->e = 0;
        } else {
            // the double-double copy of the sum for the final reduction (exact: hi + lo of a float-float)
            ms->gsum = DD{(double)total.hi + (double)total.lo, 0.0};
            // gbar = gsum / n in float-float: one Newton step on the float quotient
            const float q = __fdiv_rn(total.hi, (float)n);
            const FF r = ff_sub(total, ff_mul(FF{q, 0.f}, ff_from_double_exact(n)));
            ms->gbar_ff = ff_quick(q, __fdiv_rn(r.hi, (float)n));
            int e = 0;
            if (top[0] > 0.f) (void)frexpf(top[0], &e);
            ms->e = e;
            ms->scale = ldexpf(1.0f, -e);
        }
    }
}

// u = g - gbar (PFF: times 2^-e, exact).
template <class P>
__device__ __forceinline__ typename P::S centred(float g, const MomentState& ms) {
    if constexpr (std::is_same<P, P64>::value) return (double)g - ms.gbar;
    else {
        const FF u = ff_sub(FF{g, 0.f}, ms.gbar_ff);
        return FF{u.hi * ms.scale, u.lo * ms.scale};
    }
}

// PFF: tile sums of u.  (P64 takes them from those of g: sum of g less count x gbar, in double-double.)
__global__ void __launch_bounds__(kSigThreads) k_u_tiles(uint64_t n, const float* __restrict__ g,
                                                         const MomentState* __restrict__ ms, FF* __restrict__ tsum) {
    __shared__ FF part[kSigThreads / 32];
    const MomentState st = *ms;
    const uint64_t base = blockIdx.x * (uint64_t)kSigTile + threadIdx.x;
    FF s = FF{0.f, 0.f};
#pragma unroll
    for (int k = 0; k < kSigItems; k++) {
        const uint64_t i = base + (uint64_t)k * kSigThreads;
        if (i < n) s = ff_add(s, centred<PFF>(g[i], st));
    }
    s = warp_sum<PFF>(s);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kSigThreads / 32; w++) s = ff_add(s, part[w]);
        tsum[blockIdx.x] = s;
    }
}
__global__ void __launch_bounds__(1024) k_u_tops(uint64_t nt, FF* __restrict__ tsum) {
    FF total;
    scan_tiles<PFF>(nt, tsum, &total);
}

// u into x (the transform's input, as a real signal) and U[s] = sum of u before s, s = 0 .. n.
template <class P>
__global__ void __launch_bounds__(kSigThreads) k_center(uint64_t n, const float* __restrict__ g,
                                                        const MomentState* __restrict__ msp,
                                                        const typename P::T* __restrict__ tpre,
                                                        typename P::S* __restrict__ x, typename P::S* __restrict__ U) {
    using T = typename P::T;
    using S = typename P::S;
    using BS = cub::BlockScan<T, kSigThreads>;
    __shared__ typename BS::TempStorage tmp;
    const MomentState ms = *msp;
    const uint64_t tile = blockIdx.x * (uint64_t)kSigTile, base = tile + (uint64_t)threadIdx.x * kSigItems;
    S u[kSigItems];
    T s = P::zero();
#pragma unroll
    for (int k = 0; k < kSigItems; k++) {
        u[k] = base + k < n ? centred<P>(g[base + k], ms) : P::none();
        s = P::add_s(s, u[k]);
    }
    T ex;
    BS(tmp).ExclusiveScan(s, ex, P::zero(), SumOp<P>());
    T run = tpre[blockIdx.x];
    if constexpr (std::is_same<P, P64>::value) run = dd_add(run, dd_neg(dd_mul_d(DD{ms.gbar, 0.0}, (double)tile)));
    run = P::add(run, ex);
    if (blockIdx.x == 0 && threadIdx.x == 0) U[0] = P::none();
#pragma unroll
    for (int k = 0; k < kSigItems; k++) {
        if (base + k >= n) break;
        run = P::add_s(run, u[k]);
        x[base + k] = u[k];
        if constexpr (std::is_same<P, P64>::value) U[base + k + 1] = run.hi + run.lo;
        else U[base + k + 1] = run;
    }
}

enum Term : int { T_A = 0, T_MA = 1, T_U2 = 2, T_V2 = 3, T_U = 4, kTerms = 5 };

// Adds four terms of element t (0 .. n) to s and the fifth, U[t], to su.  uN = U[n].
// su is in double-double in both precisions, as are the prefix sums over the tiles: the window mean of a short
// L is what is left of sums of U a few 1e6 times its size (in 48 bits that was wrong by 4e-10 of it at 2^21
// bins; 713 -> 732 us there in float-float).
template <class P>
__device__ __forceinline__ void add_terms(uint64_t t, uint64_t n, const typename P::S* __restrict__ A,
                                          const typename P::S* __restrict__ U, typename P::S uN,
                                          typename P::T* s, DD& su) {
    using S = typename P::S;
    if (t > n) return;
    const S u = U[t];
    su = P64::add_s(su, P::value(u, 0));
    if (t == 0) return;
    s[T_U2] = P::add_s(s[T_U2], P::mul(u, u));  // U[t]^2, t >= 1
    if (t >= n) return;
    const S a = A[t], d = P::sub(uN, U[n - t]);
    s[T_A] = P::add_s(s[T_A], a);                              // A[t], 1 <= t < n
    s[T_MA] = P::add_s(s[T_MA], P::mul(P::of_index(t), a));    // t A[t]
    s[T_V2] = P::add_s(s[T_V2], P::mul(d, d));                 // (U[n] - U[n - t])^2
}

constexpr int kTermThreads = 256, kTermTile = 1024;

// tsum[q * nt + tile] = sum of term q over the tile.
template <class P>
__global__ void __launch_bounds__(kTermThreads) k_term_tiles(uint64_t n, uint64_t nt,
                                                             const typename P::S* __restrict__ A,
                                                             const typename P::S* __restrict__ U,
                                                             DD* __restrict__ tsum) {
    using T = typename P::T;
    __shared__ T part[T_U][kTermThreads / 32];
    __shared__ DD part_u[kTermThreads / 32];
    const typename P::S uN = U[n];
    T s[T_U];
    DD su{0.0, 0.0};
#pragma unroll
    for (int q = 0; q < T_U; q++) s[q] = P::zero();
#pragma unroll
    for (int k = 0; k < kTermTile / kTermThreads; k++)
        add_terms<P>(blockIdx.x * (uint64_t)kTermTile + k * kTermThreads + threadIdx.x, n, A, U, uN, s, su);
#pragma unroll
    for (int q = 0; q < T_U; q++) {
        const T v = warp_sum<P>(s[q]);
        if ((threadIdx.x & 31) == 0) part[q][threadIdx.x >> 5] = v;
    }
    su = warp_sum<P64>(su);
    if ((threadIdx.x & 31) == 0) part_u[threadIdx.x >> 5] = su;
    __syncthreads();
    if (threadIdx.x < T_U) {
        T v = part[threadIdx.x][0];
        for (int w = 1; w < kTermThreads / 32; w++) v = P::add(v, part[threadIdx.x][w]);
        tsum[threadIdx.x * nt + blockIdx.x] = P::sum_dd(v, 0);
    } else if (threadIdx.x == T_U) {
        DD v = part_u[0];
        for (int w = 1; w < kTermThreads / 32; w++) v = dd_add(v, part_u[w]);
        tsum[T_U * nt + blockIdx.x] = v;
    }
}

// Block q: term q's tile sums into exclusive prefix sums; total[q] = the whole.
__global__ void __launch_bounds__(1024) k_term_tops(uint64_t nt, DD* __restrict__ tsum, DD* __restrict__ total) {
    DD t;
    scan_tiles<P64>(nt, tsum + blockIdx.x * nt, &t);
    if (threadIdx.x == 0) total[blockIdx.x] = t;
}

// Windows with few positions (nw = N - L + 1 small, L close to N): the window sums F_L(j) then differ
// from one another by a small part of their size, and any formula that forms the second moment and
// subtracts the squared mean cancels (the reference's own f64 formula loses all digits there).
// These L, the last of the grid, are reduced directly: d_j = F_L(j) - F_L(0) = (U[j+L] - U[j]) - U[L]
// from the prefix sums U of the centred signal (U[0] = 0), summed with d_j^2 in double-double over the
// nw windows, and var = sum d^2 / nw - (sum d / nw)^2.  Block (p, y): part p of the windows of the
// y-th such L (one block for all the windows of an L: 116 us for 15 L of up to 65,536 windows).
template <typename UT>
__global__ void __launch_bounds__(256) k_direct_part(const uint64_t* __restrict__ grid, uint32_t first, uint64_t n,
                                                     const UT* __restrict__ U, uint64_t per_part,
                                                     DD* __restrict__ out) {
    __shared__ DD r1[8], r2[8];
    const uint64_t L = grid[first + blockIdx.y], nw = n - L + 1;
    const uint64_t a = blockIdx.x * per_part, b = min(a + per_part, nw);
    const DD uL = dd_neg(u_at<UT>(U, L));
    DD s1{0.0, 0.0}, s2{0.0, 0.0};
    for (uint64_t j = a + threadIdx.x; j < b; j += blockDim.x) {
        const DD d = dd_add(dd_add(u_at<UT>(U, j + L), dd_neg(u_at<UT>(U, j))), uL);
        s1 = dd_add(s1, d);
        s2 = dd_add(s2, dd_mul(d, d));
    }
    s1 = warp_sum<P64>(s1);
    s2 = warp_sum<P64>(s2);
    if ((threadIdx.x & 31) == 0) {
        r1[threadIdx.x >> 5] = s1;
        r2[threadIdx.x >> 5] = s2;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) {
            s1 = dd_add(s1, r1[w]);
            s2 = dd_add(s2, r2[w]);
        }
        DD* o = out + 2 * ((uint64_t)blockIdx.y * gridDim.x + blockIdx.x);
        o[0] = s1;
        o[1] = s2;
    }
}

// One block per grid point: its prefix sums (the tiles before plus the part of its own tile), then the
// final reduction and the variance subtraction in FP64.  parts > 0: grid points from `first` on take
// their variance from k_direct_part's sums.
constexpr int kPointThreads = 128;
__device__ __forceinline__ DD scaled_dd(DD a, int sc) { return DD{ldexp(a.hi, sc), ldexp(a.lo, sc)}; }
template <class P>
__global__ void __launch_bounds__(kPointThreads) k_window_moments(
    const uint64_t* __restrict__ grid, uint64_t n, uint64_t nt, const typename P::S* __restrict__ A,
    const typename P::S* __restrict__ U, const DD* __restrict__ tpre,
    const DD* __restrict__ total, const MomentState* __restrict__ msp, uint32_t first, uint32_t parts,
    const DD* __restrict__ direct, float2* __restrict__ out, double* __restrict__ mean_out,
    double* __restrict__ var_out) {
    using T = typename P::T;
    __shared__ T part[T_U][kPointThreads / 32];
    __shared__ DD part_u[2][kPointThreads / 32];
    const uint32_t i = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t L = grid[i];
    // inclusive prefix up to t = L - 1 (the t = 0 terms of A and t A are zero); UU(N-L+1) = sum of U[0 .. N-L]
    const uint64_t at_l = L - 1, at_r = n - L;
    const uint64_t tl = at_l / kTermTile, tr = at_r / kTermTile;
    const typename P::S uN = U[n];
    T s[T_U];
    DD ul{0.0, 0.0}, ur{0.0, 0.0};
#pragma unroll
    for (int q = 0; q < T_U; q++) s[q] = P::zero();
    for (uint64_t t = tl * kTermTile + threadIdx.x; t <= at_l; t += kPointThreads)
        add_terms<P>(t, n, A, U, uN, s, ul);
    for (uint64_t t = tr * kTermTile + threadIdx.x; t <= at_r; t += kPointThreads)
        ur = P64::add_s(ur, P::value(U[t], 0));
#pragma unroll
    for (int q = 0; q < T_U; q++) {
        const T v = warp_sum<P>(s[q]);
        if (lane == 0) part[q][warp] = v;
    }
    ul = warp_sum<P64>(ul);
    ur = warp_sum<P64>(ur);
    if (lane == 0) {
        part_u[0][warp] = ul;
        part_u[1][warp] = ur;
    }
    DD d1{0.0, 0.0}, d2{0.0, 0.0};
    const bool few = parts && i >= first;
    if (few && warp == 0) {
        const DD* d = direct + 2 * (uint64_t)(i - first) * parts;
        for (uint32_t p = lane; p < parts; p += 32) {
            d1 = dd_add(d1, d[2 * p]);
            d2 = dd_add(d2, d[2 * p + 1]);
        }
        d1 = warp_sum<P64>(d1);
        d2 = warp_sum<P64>(d2);
    }
    __syncthreads();
    if (threadIdx.x) return;
    const MomentState ms = *msp;
    const int e = ms.e;
    DD p[kTerms + 1];
#pragma unroll
    for (int q = 0; q <= kTerms; q++) {
        const int term = q < kTerms ? q : T_U;
        DD v = tpre[term * nt + (q < kTerms ? tl : tr)];
        for (int w = 0; w < kPointThreads / 32; w++)
            v = dd_add(v, term == T_U ? part_u[q - T_U][w] : P::sum_dd(part[q][w], 0));
        p[q] = scaled_dd(v, term == T_U ? e : 2 * e);
    }
    const double nw = (double)(n - L + 1);
    const double gbar = ms.gsum.hi / (double)n + ms.gsum.lo / (double)n;
    const double a0 = P::value(A[0], 2 * e);
    // sum_j F_L(j) = (UU(N+1) - UU(L)) - UU(N-L+1)
    const DD sf = dd_add(dd_add(scaled_dd(total[T_U], e), dd_neg(p[T_U])), dd_neg(p[kTerms]));
    const double fbar = (sf.hi + sf.lo) / nw;
    // sum_j F_L(j)^2 = L A[0] + 2 (L P0 - P1) - Q - V
    DD s2 = DD{(double)L * a0, fma((double)L, a0, -(double)L * a0)};
    const DD inner = dd_add(dd_mul_d(p[T_A], (double)L), dd_neg(p[T_MA]));
    s2 = dd_add(s2, dd_mul_d(inner, 2.0));
    s2 = dd_add(s2, dd_neg(p[T_U2]));
    s2 = dd_add(s2, dd_neg(p[T_V2]));
    const double mean = (double)L * gbar + fbar;
    double var = (s2.hi + s2.lo) / nw - fbar * fbar;
    if (!(var > 0.0)) var = 0.0;
    if (few) {  // few windows: reduced directly
        const DD m1 = dd_div_d(d1, nw), m2 = dd_div_d(d2, nw);
        const DD v = dd_add(m2, dd_neg(dd_mul(m1, m1)));
        const double scale = ldexp(1.0, e);
        var = (v.hi + v.lo) * scale * scale;
        if (!(var > 0.0)) var = 0.0;
    }
    out[i] = make_float2((float)mean, (float)var);
    if (mean_out) mean_out[i] = mean;
    if (var_out) var_out[i] = var;
}

}  // namespace rgl

using namespace rgl;

// Per-build device workspace (grown on demand) and the host twiddle table.
namespace {
struct MomentWs {
    DevBuf iv, key_a, key_b, val_a, val_b, g, totals, nz, idx, cum, cnt, fa, fb, pw, U, A, sums, state, direct, gl, tmp,
        mv;
};
std::mutex g_ws_mu;
MomentWs g_ws[16];  // one workspace per device ordinal
bool g_tw_ready[64] = {false};

// The constant tables exp(-2 pi i k / 256) of both arithmetics, once per device.
int upload_twiddles(int device) {
    if (device >= 0 && device < 64 && g_tw_ready[device]) return RGL_OK;
    double2 tw[256];
    float twf[256][4];
    for (int k = 0; k < 256; k++) {
        const long double a = -2.0L * 3.141592653589793238462643383279502884L * (long double)k / 256.0L;
        const long double v[2] = {cosl(a), sinl(a)};
        tw[k] = make_double2((double)v[0], (double)v[1]);
        for (int h = 0; h < 2; h++) {  // float-float: hi = nearest float, lo = nearest float of the remainder
            twf[k][2 * h] = (float)v[h];
            twf[k][2 * h + 1] = (float)(v[h] - (long double)twf[k][2 * h]);
        }
    }
    RGL_CUDA(cudaMemcpyToSymbol(c_tw256, tw, sizeof(tw)));
    RGL_CUDA(cudaMemcpyToSymbol(c_tw256f, twf, sizeof(twf)));
    if (device >= 0 && device < 64) g_tw_ready[device] = true;
    return RGL_OK;
}

inline unsigned blocks_for(uint64_t n) { return (unsigned)((n + 255) / 256); }

// Bit-exact reference depth signal of n intervals into ws.g (N floats).
int depth_signal_dev(MomentWs& w, const rgl_interval* h_iv, uint64_t n, uint64_t N, uint32_t bin, cudaStream_t st) {
    RGL_TRY(w.g.ensure(std::max<uint64_t>(N, 8) * 4 + 64));
    RGL_CUDA(cudaMemsetAsync(w.g.p, 0, N * 4 + 64, st));
    if (n) {
        if (n >= (1ull << 29)) return fail(RGL_ERR_INVALID_ARGUMENT, "too many intervals for one depth signal");
        const uint64_t m = 4 * n;
        RGL_TRY(w.iv.ensure(n * sizeof(rgl_interval)));
        RGL_TRY(w.key_a.ensure(m * 4));
        RGL_TRY(w.key_b.ensure(m * 4));
        RGL_TRY(w.val_a.ensure(m * 4));
        RGL_TRY(w.val_b.ensure(m * 4));
        RGL_CUDA(cudaMemcpyAsync(w.iv.p, h_iv, n * sizeof(rgl_interval), cudaMemcpyHostToDevice, st));
        k_spike_records<<<blocks_for(n), 256, 0, st>>>((uint32_t)n, w.iv.as<rgl_interval>(), (uint32_t)N, bin,
                                                        w.key_a.as<uint32_t>(), w.val_a.as<float>());
        const int bits = spike_key_bits(N);
        size_t tb = 0;
        cub::DeviceRadixSort::SortPairs(nullptr, tb, w.key_a.as<uint32_t>(), w.key_b.as<uint32_t>(), w.val_a.as<float>(),
                                        w.val_b.as<float>(), (int)m, 0, bits, st);
        RGL_TRY(w.tmp.ensure(tb + 256));
        tb = w.tmp.cap;
        RGL_CUDA(cub::DeviceRadixSort::SortPairs(w.tmp.p, tb, w.key_a.as<uint32_t>(), w.key_b.as<uint32_t>(),
                                                 w.val_a.as<float>(), w.val_b.as<float>(), (int)m, 0, bits, st));
        k_bin_sums<<<blocks_for(m), 256, 0, st>>>(m, (uint32_t)N, w.key_b.as<uint32_t>(), w.val_b.as<float>(),
                                                  w.g.as<float>());
    }
    if (N <= 1) return RGL_OK;
    const uint64_t full = N / 8;
    RGL_TRY(w.totals.ensure(full * 4 + 16));
    RGL_TRY(w.nz.ensure(full + 16));
    RGL_TRY(w.idx.ensure(full * 4 + 16));
    RGL_TRY(w.cum.ensure(full * 4 + 16));
    RGL_TRY(w.cnt.ensure(16));
    if (full) k_chunk_local<<<blocks_for(full), 256, 0, st>>>(full, w.g.as<float>(), w.totals.as<float>(), w.nz.as<uint8_t>());
    RGL_CUDA(cudaMemsetAsync(w.cnt.p, 0, 16, st));
    if (full) {
        size_t tb = 0;
        cub::DeviceSelect::Flagged(nullptr, tb, thrust::counting_iterator<uint32_t>(0), w.nz.as<uint8_t>(),
                                   w.idx.as<uint32_t>(), w.cnt.as<int>(), (int)full, st);
        RGL_TRY(w.tmp.ensure(tb + 256));
        tb = w.tmp.cap;
        RGL_CUDA(cub::DeviceSelect::Flagged(w.tmp.p, tb, thrust::counting_iterator<uint32_t>(0), w.nz.as<uint8_t>(),
                                            w.idx.as<uint32_t>(), w.cnt.as<int>(), (int)full, st));
    }
    k_carry_chain<<<1, kChainThreads, 0, st>>>(w.cnt.as<int>(), w.idx.as<uint32_t>(), w.totals.as<float>(),
                                               w.cum.as<float>(), w.g.as<float>(), N, full);
    if (full)
        k_apply_carry<<<blocks_for(full), 256, 0, st>>>(full, w.cnt.as<int>(), w.idx.as<uint32_t>(), w.cum.as<float>(),
                                                        w.g.as<float>());
    RGL_CUDA(cudaGetLastError());
    return RGL_OK;
}

template <class P, int R2, int SRC>
int fft_pass(const void* in, typename P::C* out, uint64_t H, uint64_t Ns, uint64_t n, cudaStream_t st) {
    constexpr int R = 16 * R2, kCols = 256 / R2;
    constexpr int smem = (SRC ? kCols * (R + 1) : kCols * R) * (int)sizeof(typename P::C);  // 64 to 68 KB
    RGL_CUDA(cudaFuncSetAttribute(k_fft_pass<P, R2, SRC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    k_fft_pass<P, R2, SRC><<<(unsigned)((H / R + kCols - 1) / kCols), 256, smem, st>>>(in, out, H, Ns, n);
    return RGL_OK;
}

// Transform of H packed points; the first pass reads `first` (SRC 1: a real signal of n elements, 2: the
// spectrum), the others go between w.fa and w.fb.  *result is one of the two.
template <class P, int SRC>
int fft_forward(MomentWs& w, const void* first, uint64_t H, uint64_t n, cudaStream_t st,
                typename P::C** result) {
    using C = typename P::C;
    C *dst = w.fa.as<C>(), *src = w.fb.as<C>();
    int h = 0;
    while ((1ull << h) < H) h++;
    if (h <= 4) {
        switch (h) {
            case 4: k_fft_small<P, 16, SRC><<<1, 1, 0, st>>>(first, dst, n); break;
            case 3: k_fft_small<P, 8, SRC><<<1, 1, 0, st>>>(first, dst, n); break;
            case 2: k_fft_small<P, 4, SRC><<<1, 1, 0, st>>>(first, dst, n); break;
            default: k_fft_small<P, 2, SRC><<<1, 1, 0, st>>>(first, dst, n); break;
        }
        *result = dst;
        return RGL_OK;
    }
    // radices of 2^4 to 2^8, as even as possible, the larger ones first
    const int passes = (h + 7) / 8, base = h / passes, more = h % passes;
    uint64_t Ns = 1;
    for (int p = 0; p < passes; p++) {
        const int r = base + (p < more ? 1 : 0);
        int s = RGL_OK;
        if (p == 0) {
            switch (r) {
                case 8: s = fft_pass<P, 16, SRC>(first, dst, H, Ns, n, st); break;
                case 7: s = fft_pass<P, 8, SRC>(first, dst, H, Ns, n, st); break;
                case 6: s = fft_pass<P, 4, SRC>(first, dst, H, Ns, n, st); break;
                default: s = fft_pass<P, 2, SRC>(first, dst, H, Ns, n, st); break;  // h >= 5: r >= 5
            }
        } else {
            switch (r) {
                case 8: s = fft_pass<P, 16, 0>(src, dst, H, Ns, n, st); break;
                case 7: s = fft_pass<P, 8, 0>(src, dst, H, Ns, n, st); break;
                case 6: s = fft_pass<P, 4, 0>(src, dst, H, Ns, n, st); break;
                case 5: s = fft_pass<P, 2, 0>(src, dst, H, Ns, n, st); break;
                default: s = fft_pass<P, 1, 0>(src, dst, H, Ns, n, st); break;
            }
        }
        RGL_TRY(s);
        Ns <<= r;
        std::swap(src, dst);
    }
    RGL_CUDA(cudaGetLastError());
    *result = src;
    return RGL_OK;
}

// K5-K7 for the depth signal in w.g (N bins): the moments of the L grid (G points, on the device at
// w.gl) into `table` and, where given, d_mean / d_var.
template <class P>
int moments_dev(MomentWs& w, uint64_t N, const std::vector<uint64_t>& grid, float2* table, double* d_mean,
                double* d_var, cudaStream_t st) {
    using S = typename P::S;
    using C = typename P::C;
    using T = typename P::T;
    constexpr bool kFF = std::is_same<P, PFF>::value;
    const uint32_t G = (uint32_t)grid.size();
    const uint64_t nt = (N + kSigTile - 1) / kSigTile, mt = N / kTermTile + 1;  // tiles of g and of the terms (0 .. N)
    uint64_t H = 1;  // packed points: half of the smallest power of two at or above 2 N
    while (H < N) H <<= 1;
    RGL_TRY(w.fa.ensure(H * 16));
    RGL_TRY(w.fb.ensure(H * 16));
    RGL_TRY(w.pw.ensure((H + 2) * sizeof(S)));
    RGL_TRY(w.U.ensure((N + 2) * sizeof(S)));
    RGL_TRY(w.A.ensure((N + 2) * sizeof(S)));
    RGL_TRY(w.sums.ensure(2 * nt * sizeof(T) + (kTerms * (mt + 1) + 4) * sizeof(DD)));
    RGL_TRY(w.state.ensure(sizeof(MomentState) + nt * 4 + 64));
    // windows with few positions: reduced directly, in parts of at least 2,048 windows
    const uint64_t few = std::max<uint64_t>(65536, N / 32);
    uint32_t first = G;
    while (first > 0 && N - grid[first - 1] + 1 <= few) first--;
    const uint64_t most = first < G ? N - grid[first] + 1 : 0;
    const uint32_t parts = (uint32_t)std::min<uint64_t>(64, (most + 2047) / 2048);
    RGL_TRY(w.direct.ensure(std::max<uint64_t>(1, (uint64_t)(G - first) * parts) * 2 * sizeof(DD)));
    const float* g = w.g.as<float>();
    const uint64_t* d_grid = w.gl.as<uint64_t>();
    MomentState* ms = w.state.as<MomentState>();
    float* tmax = reinterpret_cast<float*>(ms + 1);
    T* tsum = w.sums.as<T>();
    T* usum = kFF ? tsum + nt : tsum;
    DD* terms = reinterpret_cast<DD*>(tsum + 2 * nt);
    DD* totals = terms + kTerms * mt;
    S* U = w.U.as<S>();
    S* A = w.A.as<S>();
    k_g_tiles<P><<<(unsigned)nt, kSigThreads, 0, st>>>(N, g, tsum, tmax);
    k_g_tops<P><<<1, 1024, 0, st>>>(N, nt, tsum, tmax, ms);
    if constexpr (kFF) {
        k_u_tiles<<<(unsigned)nt, kSigThreads, 0, st>>>(N, g, ms, usum);
        k_u_tops<<<1, 1024, 0, st>>>(nt, usum);
    }
    S* x = A;  // the signal, read by the transform's first pass
    k_center<P><<<(unsigned)nt, kSigThreads, 0, st>>>(N, g, ms, usum, x, U);
    // K6: A[m] = Re(FFT(|FFT(u)|^2))[m] / M
    C *Z = nullptr, *Q = nullptr;
    S* pw = w.pw.as<S>();
    RGL_TRY((fft_forward<P, 1>(w, x, H, N, st, &Z)));
    k_power<P><<<blocks_for(H / 2 + 1), 256, 0, st>>>(H, Z, pw);
    RGL_TRY((fft_forward<P, 2>(w, pw, H, 0, st, &Q)));
    k_autocorr<P><<<blocks_for(H / 2 + 1), 256, 0, st>>>(H, N, Q, A);
    // K7
    k_term_tiles<P><<<(unsigned)mt, kTermThreads, 0, st>>>(N, mt, A, U, terms);
    k_term_tops<<<kTerms, 1024, 0, st>>>(mt, terms, totals);
    if (parts)
        k_direct_part<S><<<dim3(parts, G - first), 256, 0, st>>>(d_grid, first, N, U, (most + parts - 1) / parts,
                                                                 w.direct.as<DD>());
    k_window_moments<P><<<G, kPointThreads, 0, st>>>(d_grid, N, mt, A, U, terms, totals, ms, first, parts,
                                                     w.direct.as<DD>(), table, d_mean, d_var);
    RGL_CUDA(cudaGetLastError());
    return RGL_OK;
}

}  // namespace

struct rgl_moments;  // defined in stats.cu
namespace rgl {
int moments_table_ptr(rgl_moments* m, uint32_t sid, uint32_t chrom, float2** ptr, uint64_t* slots, uint64_t* n_bins,
                      int* device);
int moments_mark(rgl_moments* m, uint32_t sid, uint32_t chrom, uint64_t entries);
}  // namespace rgl

extern "C" {

int rgl_depth_signal(int device, const rgl_interval* intervals, uint64_t n, uint64_t n_bins, uint32_t bin_size,
                     float* g_out) {
    clear_error();
    if ((n && !intervals) || !g_out || bin_size == 0) return fail(RGL_ERR_INVALID_ARGUMENT, "bad arguments");
    if (n_bins * (uint64_t)bin_size > 0xFFFFFFFFull) return fail(RGL_ERR_INVALID_ARGUMENT, "n_bins * bin_size overflows u32");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return fail(RGL_ERR_NO_DEVICE, "no CUDA device");
    if (device < 0 || device >= 16 || device >= ndev) return fail(RGL_ERR_INVALID_ARGUMENT, "device ordinal out of range");
    DeviceScope scope;
    RGL_TRY(scope.enter(device));
    std::lock_guard<std::mutex> lk(g_ws_mu);
    RGL_TRY(depth_signal_dev(g_ws[device], intervals, n, n_bins, bin_size, 0));
    RGL_CUDA(cudaMemcpy(g_out, g_ws[device].g.p, n_bins * 4, cudaMemcpyDeviceToHost));
    return RGL_OK;
}

int rgl_moments_build_ex(rgl_moments* m, uint32_t sid, uint32_t chrom, const rgl_interval* intervals, uint64_t n,
                         uint32_t bin_size, uint32_t precision, double* mean_out, double* var_out) {
    clear_error();
    if (!m || (n && !intervals) || bin_size == 0) return fail(RGL_ERR_INVALID_ARGUMENT, "bad arguments");
    if (precision != RGL_MOM_FP64 && precision != RGL_MOM_FP32C)
        return fail(RGL_ERR_INVALID_ARGUMENT, "precision must be RGL_MOM_FP64 or RGL_MOM_FP32C");
    float2* table = nullptr;
    uint64_t slots = 0, N = 0;
    int device = 0;
    RGL_TRY(moments_table_ptr(m, sid, chrom, &table, &slots, &N, &device));
    if (N * (uint64_t)bin_size > 0xFFFFFFFFull) return fail(RGL_ERR_INVALID_ARGUMENT, "n_bins * bin_size overflows u32");
    if (device < 0 || device >= 16) return fail(RGL_ERR_INVALID_ARGUMENT, "device ordinal out of range");
    if (N <= 1) return moments_mark(m, sid, chrom, 0);  // moments_from_signal returns no entries
    if (N >= (1ull << 31)) return fail(RGL_ERR_INVALID_ARGUMENT, "at most 2^31 - 1 bins per chromosome");
    DeviceScope scope;
    RGL_TRY(scope.enter(device));
    std::lock_guard<std::mutex> lk(g_ws_mu);
    MomentWs& w = g_ws[device];
    cudaStream_t st = 0;
    RGL_TRY(upload_twiddles(device));
    RGL_TRY(depth_signal_dev(w, intervals, n, N, bin_size, st));
    // K7 points: the L grid of the store
    const std::vector<uint64_t> grid = moment_grid(N);
    const uint32_t G = (uint32_t)grid.size();
    if (G != slots) return fail(RGL_ERR_INVALID_ARGUMENT, "moment table size does not match the L grid");
    RGL_TRY(w.gl.ensure(G * 8ull + 64));
    RGL_CUDA(cudaMemcpyAsync(w.gl.p, grid.data(), G * 8, cudaMemcpyHostToDevice, st));
    RGL_TRY(w.mv.ensure(G * 16ull + 64));
    double* d_mean = mean_out ? w.mv.as<double>() : nullptr;
    double* d_var = var_out ? w.mv.as<double>() + G : nullptr;
    if (precision == RGL_MOM_FP32C) RGL_TRY(moments_dev<PFF>(w, N, grid, table, d_mean, d_var, st));
    else RGL_TRY(moments_dev<P64>(w, N, grid, table, d_mean, d_var, st));
    if (mean_out) RGL_CUDA(cudaMemcpyAsync(mean_out, d_mean, G * 8, cudaMemcpyDeviceToHost, st));
    if (var_out) RGL_CUDA(cudaMemcpyAsync(var_out, d_var, G * 8, cudaMemcpyDeviceToHost, st));
    RGL_CUDA(cudaStreamSynchronize(st));
    return moments_mark(m, sid, chrom, G);
}

int rgl_moments_build(rgl_moments* m, uint32_t sid, uint32_t chrom, const rgl_interval* intervals, uint64_t n,
                      uint32_t bin_size, double* mean_out, double* var_out) {
    return rgl_moments_build_ex(m, sid, chrom, intervals, n, bin_size, RGL_MOM_FP64, mean_out, var_out);
}

}  // extern "C"

// ================================================================================================
// Allocation-free depth signal.
//
// Some callers cannot allocate device memory while they call this library: code that is recording
// a CUDA graph (cudaMalloc / cudaFree are not capturable operations), hosts that route every
// device allocation through their own arena or memory pool and forbid allocations behind its back,
// and latency-critical loops that cannot afford cudaMalloc's implicit device-wide synchronisation.
// rgl_depth_signal_noalloc serves them: the same bit-exact depth signal as rgl_depth_signal, from
// device-resident intervals into a caller-provided device buffer, with all of its scratch (impulse
// records, sort buffers, per-chunk carries, CUB temporary storage) in one fixed array in this
// file.  The array is a static device variable: every GPU that loads the library holds its
// RGL_NOALLOC_SCRATCH_BYTES until the process exits.
// ================================================================================================
namespace {

constexpr uint64_t kNaMaxIv = RGL_NOALLOC_MAX_INTERVALS;
constexpr uint64_t kNaMaxBins = RGL_NOALLOC_MAX_BINS;
constexpr uint64_t kNaKeys = 4 * kNaMaxIv * 4;           // one key array (u32 x 4 records per interval)
constexpr uint64_t kNaVals = 4 * kNaMaxIv * 4;           // one value array (f32)
constexpr uint64_t kNaChunks = kNaMaxBins / 8;
constexpr uint64_t kNaOffKeyA = 0;
constexpr uint64_t kNaOffKeyB = kNaOffKeyA + kNaKeys;
constexpr uint64_t kNaOffValA = kNaOffKeyB + kNaKeys;
constexpr uint64_t kNaOffValB = kNaOffValA + kNaVals;
constexpr uint64_t kNaOffTot = kNaOffValB + kNaVals;
constexpr uint64_t kNaOffIdx = kNaOffTot + kNaChunks * 4;
constexpr uint64_t kNaOffCum = kNaOffIdx + kNaChunks * 4;
constexpr uint64_t kNaOffNz = kNaOffCum + kNaChunks * 4;
constexpr uint64_t kNaOffCnt = kNaOffNz + ((kNaChunks + 255) / 256) * 256;
constexpr uint64_t kNaOffTmp = kNaOffCnt + 256;
static_assert(kNaOffTmp < RGL_NOALLOC_SCRATCH_BYTES, "scratch layout exceeds its array");
constexpr uint64_t kNaTmpBytes = RGL_NOALLOC_SCRATCH_BYTES - kNaOffTmp;

}  // namespace

static __device__ __align__(256) unsigned char g_noalloc_scratch[RGL_NOALLOC_SCRATCH_BYTES];

namespace {
std::mutex g_na_mu;
struct NoallocSlot {
    unsigned long long ctx_id = 0;  // the context the address belongs to (0: not looked up yet)
    unsigned char* ptr = nullptr;   // device address of g_noalloc_scratch in that context
};
NoallocSlot g_na[64];

// The unique id of the calling thread's current context (cuCtxGetId, unique for the life of the
// process, so a context destroyed by cudaDeviceReset and made again gets a new one), through the
// runtime's driver entry points so that the library needs no link against libcuda.
typedef int (*CtxGetCurrentFn)(void**);
typedef int (*CtxGetIdFn)(void*, unsigned long long*);
int current_context_id(unsigned long long* id) {
    static CtxGetCurrentFn get_current = nullptr;
    static CtxGetIdFn get_id = nullptr;
    if (!get_current || !get_id) {
        void* f1 = nullptr;
        void* f2 = nullptr;
        cudaDriverEntryPointQueryResult q1{}, q2{};
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f1, cudaEnableDefault, &q1) != cudaSuccess ||
            cudaGetDriverEntryPoint("cuCtxGetId", &f2, cudaEnableDefault, &q2) != cudaSuccess || !f1 || !f2)
            return fail(RGL_ERR_DEVICE, "driver entry points cuCtxGetCurrent / cuCtxGetId are unavailable");
        get_current = reinterpret_cast<CtxGetCurrentFn>(f1);
        get_id = reinterpret_cast<CtxGetIdFn>(f2);
    }
    void* ctx = nullptr;
    if (get_current(&ctx) != 0 || !ctx) return fail(RGL_ERR_DEVICE, "no current CUDA context");
    if (get_id(ctx, id) != 0) return fail(RGL_ERR_DEVICE, "cuCtxGetId failed");
    return RGL_OK;
}

// With `device` current: the array's device address in the current context (the symbol itself is
// only a host-side stand-in), looked up on the first call and again whenever the device's context
// has changed since (after cudaDeviceReset the module is loaded anew, possibly elsewhere), and a
// check that CUB's temporary storage for the largest inputs fits.
int noalloc_setup(int device, unsigned char** out) {
    std::lock_guard<std::mutex> lk(g_na_mu);
    unsigned long long id = 0;
    RGL_TRY(current_context_id(&id));
    NoallocSlot& slot = g_na[device];
    if (slot.ctx_id != id || !slot.ptr) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess)
            return fail(RGL_ERR_DEVICE, std::string("cudaGetSymbolAddress(scratch): ") + cudaGetErrorString(e));
        size_t sort_b = 0, sel_b = 0;
        cub::DeviceRadixSort::SortPairs(nullptr, sort_b, (uint32_t*)nullptr, (uint32_t*)nullptr, (float*)nullptr,
                                        (float*)nullptr, (int)(4 * kNaMaxIv), 0, 32);
        cub::DeviceSelect::Flagged(nullptr, sel_b, thrust::counting_iterator<uint32_t>(0), (uint8_t*)nullptr,
                                   (uint32_t*)nullptr, (int*)nullptr, (int)kNaChunks);
        if (std::max(sort_b, sel_b) > kNaTmpBytes)
            return fail(RGL_ERR_UNSUPPORTED, "CUB temporary storage exceeds the reserved scratch");
        slot.ptr = static_cast<unsigned char*>(p);
        slot.ctx_id = id;
    }
    *out = slot.ptr;
    return RGL_OK;
}
}  // namespace

extern "C" int rgl_depth_signal_noalloc(int device, const rgl_interval* d_intervals, uint64_t n, uint64_t n_bins,
                                        uint32_t bin_size, float* d_g, void* stream) {
    clear_error();
    if ((n && !d_intervals) || !d_g || bin_size == 0 || n_bins == 0) return fail(RGL_ERR_INVALID_ARGUMENT, "bad arguments");
    if (n > kNaMaxIv)
        return fail(RGL_ERR_INVALID_ARGUMENT, "rgl_depth_signal_noalloc takes at most " +
                                                  std::to_string(kNaMaxIv) + " intervals (got " + std::to_string(n) + ")");
    if (n_bins > kNaMaxBins)
        return fail(RGL_ERR_INVALID_ARGUMENT, "rgl_depth_signal_noalloc takes at most " +
                                                  std::to_string(kNaMaxBins) + " bins (got " + std::to_string(n_bins) + ")");
    if (n_bins * (uint64_t)bin_size > 0xFFFFFFFFull) return fail(RGL_ERR_INVALID_ARGUMENT, "n_bins * bin_size overflows u32");
    // the chunk pass reads and writes d_g as float4, the spike pass reads the intervals as u32 words
    if (reinterpret_cast<uintptr_t>(d_g) % 16 != 0)
        return fail(RGL_ERR_INVALID_ARGUMENT, "d_g must be 16-byte aligned");
    if (reinterpret_cast<uintptr_t>(d_intervals) % 4 != 0)
        return fail(RGL_ERR_INVALID_ARGUMENT, "d_intervals must be 4-byte aligned");
    if (device < 0 || device >= 64) return fail(RGL_ERR_INVALID_ARGUMENT, "device ordinal out of range");
    DeviceScope scope;
    RGL_TRY(scope.enter(device));
    unsigned char* base = nullptr;
    RGL_TRY(noalloc_setup(device, &base));
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    uint32_t* key_a = reinterpret_cast<uint32_t*>(base + kNaOffKeyA);
    uint32_t* key_b = reinterpret_cast<uint32_t*>(base + kNaOffKeyB);
    float* val_a = reinterpret_cast<float*>(base + kNaOffValA);
    float* val_b = reinterpret_cast<float*>(base + kNaOffValB);
    float* totals = reinterpret_cast<float*>(base + kNaOffTot);
    uint32_t* idx = reinterpret_cast<uint32_t*>(base + kNaOffIdx);
    float* cum = reinterpret_cast<float*>(base + kNaOffCum);
    uint8_t* nz = base + kNaOffNz;
    int* cnt = reinterpret_cast<int*>(base + kNaOffCnt);
    void* tmp = base + kNaOffTmp;
    // the output and the compacted-chunk count start at zero; every other scratch word a call reads
    // it writes first
    RGL_CUDA(cudaMemsetAsync(d_g, 0, n_bins * 4, st));
    RGL_CUDA(cudaMemsetAsync(cnt, 0, 4, st));
    if (n) {
        const uint64_t m = 4 * n;
        k_spike_records<<<blocks_for(n), 256, 0, st>>>((uint32_t)n, d_intervals, (uint32_t)n_bins, bin_size, key_a, val_a);
        size_t tb = kNaTmpBytes;
        RGL_CUDA(cub::DeviceRadixSort::SortPairs(tmp, tb, key_a, key_b, val_a, val_b, (int)m, 0,
                                                 spike_key_bits(n_bins), st));
        k_bin_sums<<<blocks_for(m), 256, 0, st>>>(m, (uint32_t)n_bins, key_b, val_b, d_g);
    }
    if (n_bins > 1) {
        const uint64_t full = n_bins / 8;
        if (full) {
            k_chunk_local<<<blocks_for(full), 256, 0, st>>>(full, d_g, totals, nz);
            size_t tb = kNaTmpBytes;
            RGL_CUDA(cub::DeviceSelect::Flagged(tmp, tb, thrust::counting_iterator<uint32_t>(0), nz, idx, cnt,
                                                (int)full, st));
        }
        k_carry_chain<<<1, kChainThreads, 0, st>>>(cnt, idx, totals, cum, d_g, n_bins, full);
        if (full) k_apply_carry<<<blocks_for(full), 256, 0, st>>>(full, cnt, idx, cum, d_g);
    }
    RGL_CUDA(cudaGetLastError());
    return RGL_OK;
}

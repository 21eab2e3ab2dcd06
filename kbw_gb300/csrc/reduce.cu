// Reductions over the state: probabilities, sequential measurement,
// collapse, Pauli-string expectation values, dump compaction and sampling.
//
// Every reduction runs on a fixed grid and finishes in the last block to
// arrive (ticket counter, no spin-wait), so results are deterministic run to
// run.  Accumulation is FP64-grade: native double for complex128 data and
// float-float (error-free products and sums) for complex64 data, widened to
// double per thread before the block tree.
#include <float.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "../../include/kbwg.h"
#include "ff.cuh"
#include "kernels.h"
#include "sweep_dev.cuh"

namespace kbwg {

// ---- accumulators ---------------------------------------------------------
struct AccF {  // float-float running sum of products
    float hi = 0.f, lo = 0.f;
    __device__ __forceinline__ void add2(float p, float e) {
        const float s = __fadd_rn(hi, p);
        const float bb = __fsub_rn(s, hi);
        float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bb)), __fsub_rn(p, bb));
        err = __fadd_rn(err, __fadd_rn(lo, e));
        hi = __fadd_rn(s, err);
        lo = __fsub_rn(err, __fsub_rn(hi, s));
    }
    __device__ __forceinline__ void add_prod(float a, float b) {
        const float p = __fmul_rn(a, b);
        add2(p, __fmaf_rn(a, b, -p));
    }
    __device__ __forceinline__ void add_prod_neg(float a, float b) {
        const float p = __fmul_rn(a, b);
        add2(-p, -__fmaf_rn(a, b, -p));
    }
    __device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
};
struct AccD {
    double v = 0.0;
    __device__ __forceinline__ void add_prod(double a, double b) { v = __fma_rn(a, b, v); }
    __device__ __forceinline__ void add_prod_neg(double a, double b) { v = __fma_rn(-a, b, v); }
    __device__ __forceinline__ double value() const { return v; }
};
template <class T> struct AccOf;
template <> struct AccOf<float> { using type = AccF; };
template <> struct AccOf<double> { using type = AccD; };

// float-float value (products kept exactly)
struct FF {
    float hi, lo;
};

// ---- block helpers ----------------------------------------------------------
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sum over the block; the result is valid in thread 0.
__device__ double block_sum(double v) {
    __shared__ double sh[32];
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) sh[w] = v;
    __syncthreads();
    double r = 0.0;
    if (w == 0) {
        r = (lane < (int)(blockDim.x >> 5)) ? sh[lane] : 0.0;
        r = warp_sum(r);
    }
    return r;
}

// Inclusive scan over the block in a fixed order; also returns the total.
__device__ double block_inclusive_scan(double v, double *total) {
    __shared__ double wsum[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += y;
    }
    __syncthreads();
    if (lane == 31) wsum[w] = v;
    __syncthreads();
    if (w == 0) {
        const int nw = blockDim.x >> 5;
        double x = (lane < nw) ? wsum[lane] : 0.0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane < nw) wsum[lane] = x;  // inclusive warp prefix
    }
    __syncthreads();
    if (w > 0) v += wsum[w - 1];
    *total = wsum[(blockDim.x >> 5) - 1];
    return v;
}

// True in the last block to finish; partials written before are visible.
__device__ bool last_block(unsigned *ticket) {
    __shared__ bool is_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) is_last = (atomicAdd(ticket, 1u) == gridDim.x - 1);
    __syncthreads();
    return is_last;
}

// Deterministic sum of partials[b * stride + k] over b by the whole block.
__device__ double sum_partials(const double *partials, int nblocks, int stride, int k) {
    double v = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += blockDim.x) v += partials[(size_t)b * stride + k];
    return block_sum(v);
}

// A sum of floats in three parts: the errors of both upper additions are kept,
// so a few dozen float-float shares add up without another rounding.
struct f3 {
    float h, m, l;
};
__device__ __forceinline__ f3 add(const f3 &a, const f3 &b) {
    const ff::f2 h = ff::two_sum(a.h, b.h), t = ff::two_sum(a.m, b.m), m = ff::two_sum(t.h, h.l);
    return f3{h.h, m.h, ff::add(ff::add(a.l, b.l), ff::add(t.l, m.l))};
}
__device__ __forceinline__ double to_double(const f3 &a) { return (double)a.h + ((double)a.m + (double)a.l); }

// Sums of up to 32 terms at once.  share(k): this thread's of term k; lane k
// returns the warp's sum of term k.  Halving exchange: 31 additions instead of
// 5 per term, and no FP64 instruction: a double tree over 32 terms took 19 us
// of a 25 us launch on GB300's FP64 pipe.  In three parts: a float-float tree
// rounds to 48 bits where the warps' sums average out least (12 qubits, rms
// error of a string without flips 3.5e-16 with a double tree, 6.9e-16 with
// that one).
template <class F>
__device__ __forceinline__ f3 warp_sum_terms(F &&share) {
    const int lane = threadIdx.x & 31;
    const bool top = (lane & 16) != 0;
    f3 t[kMaxTerms / 2];
#pragma unroll
    for (int i = 0; i < kMaxTerms / 2; i++) {
        const f3 a = share(i), b = share(i + 16), keep = top ? b : a, send = top ? a : b;
        t[i] = add(keep, f3{__shfl_xor_sync(0xffffffffu, send.h, 16), __shfl_xor_sync(0xffffffffu, send.m, 16),
                            __shfl_xor_sync(0xffffffffu, send.l, 16)});
    }
#pragma unroll
    for (int w = 8; w > 0; w >>= 1) {
        const bool up = (lane & w) != 0;
#pragma unroll
        for (int i = 0; i < w; i++) {
            const f3 keep = up ? t[i + w] : t[i], send = up ? t[i] : t[i + w];
            t[i] = add(keep, f3{__shfl_xor_sync(0xffffffffu, send.h, w), __shfl_xor_sync(0xffffffffu, send.m, w),
                                __shfl_xor_sync(0xffffffffu, send.l, w)});
        }
    }
    return t[0];
}

// The grid's sums of nt terms into rs.result: lane k of every warp holds its
// warp's sum of term k.  Fixed order (warps, then blocks by warp of the last
// block), so deterministic.  256 threads; every thread calls it.
__device__ void finish_terms(double v, uint32_t nt, const ReduceScratch &rs) {
    __shared__ double sh[kReduceThreads / 32][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    sh[w][lane] = v;
    __syncthreads();
    if (w == 0 && lane < (int)nt) {
        double t = 0.0;
        for (int j = 0; j < kReduceThreads / 32; j++) t += sh[j][lane];
        rs.partials[(size_t)blockIdx.x * kMaxTerms + lane] = t;
    }
    if (last_block(rs.ticket)) {
        double t = 0.0;
        if (lane < (int)nt)
            for (unsigned b = (unsigned)w; b < gridDim.x; b += kReduceThreads / 32)
                t += __ldcg(rs.partials + (size_t)b * kMaxTerms + lane);
        sh[w][lane] = t;
        __syncthreads();
        if (w == 0 && lane < (int)nt) {
            double r = 0.0;
            for (int j = 0; j < kReduceThreads / 32; j++) r += sh[j][lane];
            rs.result[lane] = r;
        }
        if (threadIdx.x == 0) *rs.ticket = 0;
    }
}

__device__ __forceinline__ uint64_t insert_zero(uint64_t i, uint32_t m) {
    const uint64_t low = (1ull << m) - 1;
    return ((i & ~low) << 1) | (i & low);
}

// Insert zero bits at every set position of M (ascending).
__device__ __forceinline__ uint64_t insert_zeros(uint64_t i, uint64_t M) {
    while (M) {
        const uint32_t m = __ffsll((long long)M) - 1;
        M &= M - 1;
        i = insert_zero(i, m);
    }
    return i;
}

// rand's UniformFloat::new(0, total) scale rule (largest draw 1 - 2^-52).
__host__ __device__ inline double uniform_scale(double total) {
    const double max_rand = 1.0 - DBL_EPSILON;
    double scale = total;
#ifdef __CUDA_ARCH__
    while (__dmul_rn(scale, max_rand) >= total) scale = __longlong_as_double(__double_as_longlong(scale) - 1);
#else
    while (scale * max_rand >= total) {
        union {
            double d;
            uint64_t u;
        } x;
        x.d = scale;
        x.u -= 1;
        scale = x.d;
    }
#endif
    return scale;
}

// ---- masked norm / p1 -------------------------------------------------------
template <class T>
__device__ __forceinline__ double masked_norm_body(const cx<T> *__restrict__ st, uint64_t count, uint64_t M,
                                                   uint64_t V) {
    typename AccOf<T>::type acc;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (; i + 3 * stride < count; i += 4 * stride) {
        cx<T> a[4];
#pragma unroll
        for (int u = 0; u < 4; u++) a[u] = st[insert_zeros(i + u * stride, M) | V];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            acc.add_prod(a[u].re, a[u].re);
            acc.add_prod(a[u].im, a[u].im);
        }
    }
    for (; i < count; i += stride) {
        const cx<T> a = st[insert_zeros(i, M) | V];
        acc.add_prod(a.re, a.re);
        acc.add_prod(a.im, a.im);
    }
    return block_sum(acc.value());
}

template <class T>
__global__ void __launch_bounds__(kReduceThreads)
    k_masked_norm(const cx<T> *__restrict__ st, uint64_t count, uint64_t M, uint64_t V, ReduceScratch rs) {
    const double v = masked_norm_body<T>(st, count, M, V);
    if (threadIdx.x == 0) rs.partials[blockIdx.x] = v;
    if (last_block(rs.ticket)) {
        const double t = sum_partials(rs.partials, gridDim.x, 1, 0);
        if (threadIdx.x == 0) {
            rs.result[0] = t;
            *rs.ticket = 0;
        }
    }
}

template <class T>
cudaError_t launch_masked_norm(const void *st, uint32_t n, uint64_t M, uint64_t V, const ReduceScratch &rs,
                               cudaStream_t s) {
    const uint64_t count = 1ull << (n - __builtin_popcountll(M));
    k_masked_norm<T><<<kReduceBlocks, kReduceThreads, 0, s>>>((const cx<T> *)st, count, M, V, rs);
    count_launch();
    return cudaGetLastError();
}

// (re^2, im^2) of an amplitude as packed products and their errors.
__device__ __forceinline__ ff2::v2 prob_square(float2 h, float2 l) {
    const float2 p = ff2::mul(h, h);
    return ff2::v2{p, ff2::fma(l, h, ff2::fma(h, l, ff2::fma(h, h, ff2::neg(p))))};
}
__device__ __forceinline__ ff2::v2 prob_square(float4 f) {  // re.hi, im.hi, re.lo, im.lo
    return prob_square(make_float2(f.x, f.y), make_float2(f.z, f.w));
}
__device__ __forceinline__ ff2::v2 prob_square(cx<double> a) {
    const ff::f2 re = ff::from_double(a.re), im = ff::from_double(a.im);
    return prob_square(make_float2(re.h, im.h), make_float2(re.l, im.l));
}
__device__ __forceinline__ ff2::v2 prob_square(cx<float> a) {
    const float2 h = make_float2(a.re, a.im), p = ff2::mul(h, h);
    return ff2::v2{p, ff2::fma(h, h, ff2::neg(p))};
}
// (|a|^2, |b|^2) from their squares, in float-float.
__device__ __forceinline__ ff2::v2 prob_pair(ff2::v2 a, ff2::v2 b) {
    const ff2::v2 t = ff2::two_sum(make_float2(a.h.x, b.h.x), make_float2(a.h.y, b.h.y));
    const float2 e = ff2::add(make_float2(a.l.x, b.l.x), make_float2(a.l.y, b.l.y));
    return ff2::fast_two_sum(t.h, ff2::add(t.l, e));
}

// The same over the float-float resident form of a complex128 state
// (re.hi, im.hi, re.lo, im.lo per amplitude): |a|^2 as a float-float dot
// product, summed per thread in float-float (FP32-pipe work), then in binary64.
__device__ __forceinline__ double masked_norm_body_ff(const float4 *__restrict__ st, uint64_t count, uint64_t M,
                                                      uint64_t V) {
    // four loads in flight per thread and two sums, packed; the last four
    // guarded, where one by one they waited for memory up to three times
    // (24-qubit p1, 128 MiB read: 32.1 -> 30.2 us, the bytes alone 20)
    ff2::v2 acc{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += 4 * stride) {
        float4 f[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint64_t x = i + u * stride;
            f[u] = x < count ? st[insert_zeros(x, M) | V] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        acc = ff2::add(acc, ff2::add(prob_pair(prob_square(f[0]), prob_square(f[2])),
                                     prob_pair(prob_square(f[1]), prob_square(f[3]))));
    }
    const ff::f2 t = ff::add(ff::f2{acc.h.x, acc.l.x}, ff::f2{acc.h.y, acc.l.y});
    return block_sum((double)t.h + (double)t.l);
}

__global__ void __launch_bounds__(kReduceThreads)
    k_masked_norm_ff(const float4 *__restrict__ st, uint64_t count, uint64_t M, uint64_t V, ReduceScratch rs) {
    const double v = masked_norm_body_ff(st, count, M, V);
    if (threadIdx.x == 0) rs.partials[blockIdx.x] = v;
    if (last_block(rs.ticket)) {
        const double t = sum_partials(rs.partials, gridDim.x, 1, 0);
        if (threadIdx.x == 0) {
            rs.result[0] = t;
            *rs.ticket = 0;
        }
    }
}

cudaError_t launch_masked_norm_ff(const void *st, uint32_t n, uint64_t M, uint64_t V, const ReduceScratch &rs,
                                  cudaStream_t s) {
    const uint64_t count = 1ull << (n - __builtin_popcountll(M));
    k_masked_norm_ff<<<kReduceBlocks, kReduceThreads, 0, s>>>((const float4 *)st, count, M, V, rs);
    count_launch();
    return cudaGetLastError();
}

// ---- distance between two states ----------------------------------------------
// partials: sum |a - b|^2 and sum |b|^2 (two values per block).
template <class T>
__global__ void __launch_bounds__(kReduceThreads)
    k_distance(const cx<T> *__restrict__ a, const cx<T> *__restrict__ b, uint64_t count, ReduceScratch rs) {
    typename AccOf<T>::type d, nb;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += stride) {
        const cx<T> x = a[i], y = b[i];
        const T dr = x.re - y.re, di = x.im - y.im;
        d.add_prod(dr, dr);
        d.add_prod(di, di);
        nb.add_prod(y.re, y.re);
        nb.add_prod(y.im, y.im);
    }
    const double vd = block_sum(d.value());
    const double vn = block_sum(nb.value());
    if (threadIdx.x == 0) {
        rs.partials[2 * blockIdx.x] = vd;
        rs.partials[2 * blockIdx.x + 1] = vn;
    }
    if (last_block(rs.ticket)) {
        const double td = sum_partials(rs.partials, gridDim.x, 2, 0);
        const double tn = sum_partials(rs.partials, gridDim.x, 2, 1);
        if (threadIdx.x == 0) {
            rs.result[0] = td;
            rs.result[1] = tn;
            *rs.ticket = 0;
        }
    }
}

template <class T>
cudaError_t launch_distance(const void *a, const void *b, uint32_t n, const ReduceScratch &rs, cudaStream_t s) {
    k_distance<T><<<kReduceBlocks, kReduceThreads, 0, s>>>((const cx<T> *)a, (const cx<T> *)b, 1ull << n, rs);
    count_launch();
    return cudaGetLastError();
}
template cudaError_t launch_distance<float>(const void *, const void *, uint32_t, const ReduceScratch &, cudaStream_t);
template cudaError_t launch_distance<double>(const void *, const void *, uint32_t, const ReduceScratch &, cudaStream_t);

// partials: Re<a|b>, Im<a|b>, <a|a>, <b|b> (four values per block), either
// precision on either side, accumulated in FP64.
template <class TA, class TB>
__global__ void __launch_bounds__(kReduceThreads)
    k_overlap(const cx<TA> *__restrict__ a, const cx<TB> *__restrict__ b, uint64_t count, ReduceScratch rs) {
    AccD re, im, na, nb;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += stride) {
        const cx<TA> x = a[i];
        const cx<TB> y = b[i];
        const double ar = x.re, ai = x.im, br = y.re, bi = y.im;
        re.add_prod(ar, br);  // conj(a) b = (ar br + ai bi) + i (ar bi - ai br)
        re.add_prod(ai, bi);
        im.add_prod(ar, bi);
        im.add_prod_neg(ai, br);
        na.add_prod(ar, ar);
        na.add_prod(ai, ai);
        nb.add_prod(br, br);
        nb.add_prod(bi, bi);
    }
    const double v0 = block_sum(re.value());
    const double v1 = block_sum(im.value());
    const double v2 = block_sum(na.value());
    const double v3 = block_sum(nb.value());
    if (threadIdx.x == 0) {
        rs.partials[4 * blockIdx.x] = v0;
        rs.partials[4 * blockIdx.x + 1] = v1;
        rs.partials[4 * blockIdx.x + 2] = v2;
        rs.partials[4 * blockIdx.x + 3] = v3;
    }
    if (last_block(rs.ticket)) {
        double t[4];
        for (int k = 0; k < 4; k++) t[k] = sum_partials(rs.partials, gridDim.x, 4, k);
        if (threadIdx.x == 0) {
            for (int k = 0; k < 4; k++) rs.result[k] = t[k];
            *rs.ticket = 0;
        }
    }
}

cudaError_t launch_overlap(const void *a, int prec_a, const void *b, int prec_b, uint32_t n, const ReduceScratch &rs,
                           cudaStream_t s) {
    const uint64_t count = 1ull << n;
    if (prec_a && prec_b)
        k_overlap<double, double><<<kReduceBlocks, kReduceThreads, 0, s>>>((const cx<double> *)a,
                                                                           (const cx<double> *)b, count, rs);
    else if (prec_a)
        k_overlap<double, float><<<kReduceBlocks, kReduceThreads, 0, s>>>((const cx<double> *)a,
                                                                          (const cx<float> *)b, count, rs);
    else if (prec_b)
        k_overlap<float, double><<<kReduceBlocks, kReduceThreads, 0, s>>>((const cx<float> *)a,
                                                                          (const cx<double> *)b, count, rs);
    else
        k_overlap<float, float><<<kReduceBlocks, kReduceThreads, 0, s>>>((const cx<float> *)a, (const cx<float> *)b,
                                                                         count, rs);
    count_launch();
    return cudaGetLastError();
}

// ---- sequential measurement step ------------------------------------------
// QubitManager::do_measure's decision for one qubit (src/quantum_execution.rs:278-287)
// from s1, the weight of its |1> side among the outcomes so far; by one thread.
template <class T>
__device__ __forceinline__ void measure_decide(MeasureCtl *ctl, uint32_t step, uint64_t bit, double s1) {
    const double p1 = __dmul_rn(s1, ctl->scale2);
    double p0 = __dsub_rn(1.0, p1);
    if (!(p0 > 0.0)) p0 = 0.0;
    const double total = __dadd_rn(p0, p1);
    const double chosen = __dmul_rn(ctl->draws[step], uniform_scale(total));
    const int r = (p0 <= chosen) ? 1 : 0;
    double prob = r ? p1 : p0;
    if (!(prob > DBL_MIN)) prob = DBL_MIN;
    const double p = 1.0 / sqrt(prob);
    const double pf = (double)(T)p;
    ctl->p[step] = p;
    ctl->scale2 = __dmul_rn(__dmul_rn(ctl->scale2, pf), pf);
    ctl->M = ctl->M | bit;
    ctl->V = ctl->V | (r ? bit : 0ull);
    ctl->result |= (uint64_t)r << step;
    ctl->steps = step + 1;
}

template <class T, bool kFF>
__device__ __forceinline__ double measure_norm(const void *__restrict__ st, uint32_t n, uint64_t M, uint64_t V) {
    const uint64_t count = 1ull << (n - __popcll(M));
    if constexpr (kFF) return masked_norm_body_ff((const float4 *)st, count, M, V);
    else return masked_norm_body<T>((const cx<T> *)st, count, M, V);
}

template <class T, bool kFF = false>
__global__ void __launch_bounds__(kReduceThreads)
    k_measure_step(const void *__restrict__ st, uint32_t n, MeasureCtl *ctl, uint32_t step, ReduceScratch rs) {
    const uint64_t bit = 1ull << ctl->qubit[step];
    const double v = measure_norm<T, kFF>(st, n, ctl->M | bit, ctl->V | bit);
    if (threadIdx.x == 0) rs.partials[blockIdx.x] = v;
    if (last_block(rs.ticket)) {
        const double s1 = sum_partials(rs.partials, gridDim.x, 1, 0);
        if (threadIdx.x == 0) {
            measure_decide<T>(ctl, step, bit, s1);
            *rs.ticket = 0;
        }
    }
}

// Steps [step, steps) by one block: once few amplitudes are left, a step is
// shorter than its launch (24 qubits: 14 of 24 steps, 13 us each before).
template <class T, bool kFF>
__global__ void __launch_bounds__(kReduceThreads)
    k_measure_tail(const void *__restrict__ st, uint32_t n, MeasureCtl *ctl, uint32_t step, uint32_t steps) {
    for (; step < steps; step++) {
        const uint64_t bit = 1ull << ctl->qubit[step];
        const double s1 = measure_norm<T, kFF>(st, n, ctl->M | bit, ctl->V | bit);
        __syncthreads();
        if (threadIdx.x == 0) measure_decide<T>(ctl, step, bit, s1);
        __syncthreads();
    }
}

// Amplitudes a step reads below which one block takes the remaining steps.
constexpr uint64_t kMeasureTail = 1ull << 12;

template <class T, bool kFF>
static cudaError_t measure_steps(const void *st, uint32_t n, MeasureCtl *ctl, uint32_t steps, const ReduceScratch &rs,
                                 cudaStream_t s) {
    for (uint32_t k = 0; k < steps; k++) {
        const uint64_t count = 1ull << (n - (k + 1));  // the qubits are distinct
        if (count <= kMeasureTail) {
            k_measure_tail<T, kFF><<<1, kReduceThreads, 0, s>>>(st, n, ctl, k, steps);
            count_launch();
            return cudaGetLastError();
        }
        const unsigned grid = (unsigned)std::min<uint64_t>(kReduceBlocks, count / (4 * kReduceThreads));
        k_measure_step<T, kFF><<<grid, kReduceThreads, 0, s>>>(st, n, ctl, k, rs);
        count_launch();
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

template <class T>
cudaError_t launch_measure_steps(const void *st, uint32_t n, MeasureCtl *ctl, uint32_t steps, const ReduceScratch &rs,
                                 cudaStream_t s) {
    return measure_steps<T, false>(st, n, ctl, steps, rs, s);
}

cudaError_t launch_measure_steps_ff(const void *st, uint32_t n, MeasureCtl *ctl, uint32_t steps,
                                    const ReduceScratch &rs, cudaStream_t s) {
    return measure_steps<double, true>(st, n, ctl, steps, rs, s);
}

// ---- collapse -----------------------------------------------------------------
template <class T>
__global__ void __launch_bounds__(256)
    k_collapse(cx<T> *__restrict__ st, uint64_t ns, const MeasureCtl *ctl, uint64_t M, uint64_t V, double p) {
    __shared__ T pf[64];
    __shared__ uint64_t sM, sV;
    __shared__ uint32_t nf;
    if (threadIdx.x == 0) {
        if (ctl) {
            sM = ctl->M;
            sV = ctl->V;
            nf = ctl->steps;
        } else {
            sM = M;
            sV = V;
            nf = 1;
        }
    }
    if (threadIdx.x < 64) pf[threadIdx.x] = ctl ? (T)ctl->p[threadIdx.x] : (T)p;
    __syncthreads();
    const uint64_t m = sM, v = sV;
    const uint32_t k = nf;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; s < ns; s += stride) {
        cx<T> a;
        if ((s & m) == v) {
            a = st[s];
            for (uint32_t j = 0; j < k; j++) {  // one multiply per collapse, in order
                a.re = xmul(a.re, pf[j]);
                a.im = xmul(a.im, pf[j]);
            }
        } else {
            a.re = (T)0;
            a.im = (T)0;
        }
        st[s] = a;
    }
}

// The collapse of a float-float resident state: each kept amplitude's parts
// times the binary64 factors 1/sqrt(P) in float-float, one per collapse, in
// order.
__global__ void __launch_bounds__(256)
    k_collapse_ff(float4 *__restrict__ st, uint64_t ns, const MeasureCtl *ctl, uint64_t M, uint64_t V, double p) {
    __shared__ float ph[64], pl[64];
    __shared__ uint64_t sM, sV;
    __shared__ uint32_t nf;
    if (threadIdx.x == 0) {
        if (ctl) {
            sM = ctl->M;
            sV = ctl->V;
            nf = ctl->steps;
        } else {
            sM = M;
            sV = V;
            nf = 1;
        }
    }
    if (threadIdx.x < 64) {
        const ff::f2 f = ff::split_constant(ctl ? ctl->p[threadIdx.x] : p);
        ph[threadIdx.x] = f.h;
        pl[threadIdx.x] = f.l;
    }
    __syncthreads();
    const uint64_t m = sM, v = sV;
    const uint32_t k = nf;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; s < ns; s += stride) {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
        if ((s & m) == v) {
            a = st[s];
            ff::f2 re{a.x, a.z}, im{a.y, a.w};
            for (uint32_t j = 0; j < k; j++) {
                const ff::f2 f{ph[j], pl[j]};
                re = ff::mul(re, f);
                im = ff::mul(im, f);
            }
            a = make_float4(re.h, im.h, re.l, im.l);
        }
        st[s] = a;
    }
}

cudaError_t launch_collapse_ff(void *st, uint32_t n, const MeasureCtl *ctl, uint64_t M, uint64_t V, double p,
                               cudaStream_t s) {
    const uint64_t ns = 1ull << n;
    uint64_t g = (ns + 255) / 256;
    if (g > 152 * 16) g = 152 * 16;
    k_collapse_ff<<<(unsigned)g, 256, 0, s>>>((float4 *)st, ns, ctl, M, V, p);
    count_launch();
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_collapse(void *st, uint32_t n, const MeasureCtl *ctl, uint64_t M, uint64_t V, double p,
                            cudaStream_t s) {
    const uint64_t ns = 1ull << n;
    uint64_t g = (ns + 255) / 256;
    if (g > 152 * 16) g = 152 * 16;
    k_collapse<T><<<(unsigned)g, 256, 0, s>>>((cx<T> *)st, ns, ctl, M, V, p);
    count_launch();
    return cudaGetLastError();
}

// ---- Pauli strings ------------------------------------------------------------
// <psi|P|psi> with P = i^{nY} X^x Z^z (per qubit).  For x == 0 the sum is
// sum_s (-1)^{|s & z|} |a_s|^2.  For x != 0 each pair (s, s^x) with bit h
// (the highest of x) clear contributes +-2 (-1)^{|s & z|} Re or Im of
// conj(a_s) a_{s^x}; the host folds i^{nY} and (-1)^{|x & z|} into `factor`
// and `use_im`.
template <class T>
__global__ void __launch_bounds__(kReduceThreads)
    k_pauli_group(const cx<T> *__restrict__ st, uint32_t n, PauliGroup g, ReduceScratch rs) {
    typename AccOf<T>::type acc[kMaxTerms];
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint32_t nt = g.nterms;
    if (g.x == 0) {
        const uint64_t count = 1ull << n;
        for (uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; s < count; s += stride) {
            const cx<T> a = st[s];
#pragma unroll
            for (int k = 0; k < kMaxTerms; k++) {
                if (k < (int)nt) {
                    if ((__popcll(s & g.z[k]) & 1) ^ (g.factor[k] < 0)) {
                        acc[k].add_prod_neg(a.re, a.re);
                        acc[k].add_prod_neg(a.im, a.im);
                    } else {
                        acc[k].add_prod(a.re, a.re);
                        acc[k].add_prod(a.im, a.im);
                    }
                }
            }
        }
    } else {
        const uint32_t h = 63 - __clzll((long long)g.x);
        const uint64_t count = 1ull << (n - 1);
        for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += stride) {
            const uint64_t s = insert_zero(i, h);
            const cx<T> a = st[s], b = st[s ^ g.x];
#pragma unroll
            for (int k = 0; k < kMaxTerms; k++) {
                if (k < (int)nt) {
                    const bool neg = (__popcll(s & g.z[k]) & 1) ^ (g.factor[k] < 0);
                    // Re(conj(a) b) = a.re b.re + a.im b.im ; Im = a.re b.im - a.im b.re
                    if (!g.use_im[k]) {
                        if (neg) {
                            acc[k].add_prod_neg(a.re, b.re);
                            acc[k].add_prod_neg(a.im, b.im);
                        } else {
                            acc[k].add_prod(a.re, b.re);
                            acc[k].add_prod(a.im, b.im);
                        }
                    } else {
                        if (neg) {
                            acc[k].add_prod_neg(a.re, b.im);
                            acc[k].add_prod(a.im, b.re);
                        } else {
                            acc[k].add_prod(a.re, b.im);
                            acc[k].add_prod_neg(a.im, b.re);
                        }
                    }
                }
            }
        }
    }
#pragma unroll
    for (int k = 0; k < kMaxTerms; k++) {
        if (k < (int)nt) {
            const double f = fabs(g.factor[k]);
            const double v = block_sum(acc[k].value() * f);
            if (threadIdx.x == 0) rs.partials[(size_t)blockIdx.x * kMaxTerms + k] = v;
        }
    }
    if (last_block(rs.ticket)) {
        for (int k = 0; k < (int)nt; k++) {
            const double t = sum_partials(rs.partials, gridDim.x, kMaxTerms, k);
            if (threadIdx.x == 0) rs.result[k] = t;
        }
        if (threadIdx.x == 0) *rs.ticket = 0;
    }
}

// The pairs of a register below one tile, a block per string: products as
// k_pauli_group forms them, summed in binary64, all strings in one launch (an
// energy call on 9 qubits with 36 such strings: a launch of 608 blocks per flip
// mask 0.83 ms, this one 0.46 ms).
template <class T>
__global__ void __launch_bounds__(kReduceThreads)
    k_pauli_small(const cx<T> *__restrict__ st, uint32_t n, const __grid_constant__ PauliSmall p, double *result) {
    const int k = (int)blockIdx.x;
    const uint64_t x = p.x[k], z = p.z[k];
    const bool im = p.use_im[k] != 0, minus = p.factor[k] < 0;
    const uint32_t h = 63 - __clzll((long long)x);
    const uint64_t count = 1ull << (n - 1);
    double sum = 0.0;
    for (uint64_t i = threadIdx.x; i < count; i += blockDim.x) {
        const uint64_t s = insert_zero(i, h);
        const cx<T> a = st[s], b = st[s ^ x];
        typename AccOf<T>::type acc;
        const T re = (__popcll(s & z) & 1) ^ minus ? -a.re : a.re, ai = (__popcll(s & z) & 1) ^ minus ? -a.im : a.im;
        // Re(conj(a) b) = a.re b.re + a.im b.im ; Im = a.re b.im - a.im b.re
        acc.add_prod(re, im ? b.im : b.re);
        acc.add_prod(im ? -ai : ai, im ? b.re : b.im);
        sum += acc.value();
    }
    const double v = block_sum(sum * fabs(p.factor[k]));
    if (threadIdx.x == 0) result[k] = v;
}

template <class T>
cudaError_t launch_pauli_small(const void *st, uint32_t n, const PauliSmall &p, const ReduceScratch &rs, cudaStream_t s) {
    k_pauli_small<T><<<p.nterms, kReduceThreads, 0, s>>>((const cx<T> *)st, n, p, rs.result);
    count_launch();
    return cudaGetLastError();
}

// Diagonal groups (x == 0) with a Walsh transform.  A warp reads 512
// consecutive amplitudes s = b + lane + 32u (u = 0..15, coalesced), so
// (-1)^{|s & z|} = (-1)^{|(b | lane) & z|} * (-1)^{|u & zu|}, zu = (z >> 5) & 15.
// Each thread forms the 16-point Walsh-Hadamard transform W of its
// probabilities p_u (64 adds) and every term adds +-W[zu]: about 4 + nt/16
// additions per amplitude instead of nt.  Two amplitudes (u, u + 8) and two
// terms share each packed instruction; a run's 32 term parities of b come from
// one popcount per lane and a ballot: bound by instruction issue, 27 float-float
// terms at 27 qubits 739 -> 572 us (reading the state alone 316).
// Probabilities and sums are
// float-float: error-free products of the complex64 parts, and for complex128
// a float-float dot product of the amplitude split into float-float (binary64
// storage) or read as is (the float-float resident form) -- FP32-pipe work
// instead of GB300's slow FP64 pipe, ~2^-48 relative per operation.
constexpr int kDiagRun = 16;                   // amplitudes per thread per run
constexpr int kDiagWarpSpan = 32 * kDiagRun;  // 512 consecutive amplitudes per warp

template <class T, bool kFF>
__global__ void __launch_bounds__(kReduceThreads, 2)
    k_pauli_diag(const void *__restrict__ st, uint32_t n, PauliGroup g, ReduceScratch rs) {
    using Load = typename pick_t<kFF, float4, cx<T>>::type;
    __shared__ float wh[kReduceThreads / 32][kDiagRun][32], wl[kReduceThreads / 32][kDiagRun][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t nt = g.nterms;
    constexpr int H = kDiagRun / 2;
    ff2::v2 acc[kMaxTerms / 2];  // terms 2k, 2k + 1
    uint32_t lanepar = 0;  // bit k: parity of (lane & z_k) xor the term's sign
    uint64_t zlane = 0;    // mask of term `lane`
#pragma unroll
    for (int k = 0; k < kMaxTerms; k++) {
        if (!(k & 1)) acc[k / 2] = ff2::v2{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        if (k < (int)nt) {
            lanepar |= (uint32_t)((__popc((uint32_t)lane & (uint32_t)g.z[k]) & 1) ^ (g.factor[k] < 0)) << k;
            if (lane == k) zlane = g.z[k];
        }
    }
    const uint64_t runs = (1ull << n) / kDiagWarpSpan;
    const uint64_t wstride = (uint64_t)gridDim.x * (blockDim.x >> 5);
    for (uint64_t r = (uint64_t)blockIdx.x * (blockDim.x >> 5) + w; r < runs; r += wstride) {
        const uint64_t b = r * kDiagWarpSpan;
        const Load *src = reinterpret_cast<const Load *>(st) + b + lane;
        ff2::v2 p[H];  // amplitudes u and u + H
#pragma unroll
        for (int u = 0; u < H; u++) p[u] = prob_pair(prob_square(src[32 * u]), prob_square(src[32 * (u + H)]));
#pragma unroll
        for (int h = 1; h < H; h <<= 1) {
#pragma unroll
            for (int u = 0; u < H; u++) {
                if (u & h) continue;
                const ff2::v2 x = p[u], y = p[u | h];
                p[u] = ff2::add(x, y);
                p[u | h] = ff2::sub(x, y);
            }
        }
#pragma unroll
        for (int u = 0; u < H; u++) {
            const ff2::v2 t = ff2::add(ff2::v2{make_float2(p[u].h.x, p[u].h.x), make_float2(p[u].l.x, p[u].l.x)},
                                       ff2::v2{make_float2(p[u].h.y, -p[u].h.y), make_float2(p[u].l.y, -p[u].l.y)});
            wh[w][u][lane] = t.h.x;
            wl[w][u][lane] = t.l.x;
            wh[w][u + H][lane] = t.h.y;
            wl[w][u + H][lane] = t.l.y;
        }
        // bit k: the sign of term k at this thread's amplitudes
        const uint32_t neg = __ballot_sync(0xffffffffu, __popcll(b & zlane) & 1) ^ lanepar;
        __syncwarp();
#pragma unroll
        for (int k = 0; k < kMaxTerms; k += 2) {
            if (k < (int)nt) {  // (a term beyond the last adds what nobody reads)
                const int i0 = (int)(g.z[k] >> 5) & 15, i1 = (int)(g.z[k + 1] >> 5) & 15;
                const uint32_t s0 = (neg << (31 - k)) & 0x80000000u, s1 = (neg << (30 - k)) & 0x80000000u;
                const auto at = [](float x, uint32_t s) { return __uint_as_float(__float_as_uint(x) ^ s); };
                acc[k / 2] = ff2::add(acc[k / 2], ff2::v2{make_float2(at(wh[w][i0][lane], s0), at(wh[w][i1][lane], s1)),
                                                          make_float2(at(wl[w][i0][lane], s0), at(wl[w][i1][lane], s1))});
            }
        }
        __syncwarp();
    }
    const f3 sum = warp_sum_terms([&](int k) {
        const ff2::v2 &a = acc[k / 2];
        return (k & 1) ? f3{a.h.y, a.l.y, 0.f} : f3{a.h.x, a.l.x, 0.f};
    });
    finish_terms(to_double(sum), nt, rs);
}

template <class T>
cudaError_t launch_pauli_group(const void *st, uint32_t n, const PauliGroup &g, const ReduceScratch &rs,
                               cudaStream_t s, bool ff_resident) {
    if (ff_resident && !(sizeof(T) == 8 && g.x == 0 && (1ull << n) >= (uint64_t)kDiagWarpSpan))
        return cudaErrorInvalidValue;  // (only the diagonal form reads the float-float resident state)
    if (g.x == 0 && (1ull << n) >= (uint64_t)kDiagWarpSpan) {
        // no block without a run of amplitudes: their tails would only queue up
        const uint64_t want = ((1ull << n) / kDiagWarpSpan + kReduceThreads / 32 - 1) / (kReduceThreads / 32);
        const unsigned grid = (unsigned)std::min<uint64_t>(want, (uint64_t)kReduceBlocks);
        if constexpr (sizeof(T) == 8) {
            if (ff_resident)
                k_pauli_diag<T, true><<<grid, kReduceThreads, 0, s>>>(st, n, g, rs);
            else
                k_pauli_diag<T, false><<<grid, kReduceThreads, 0, s>>>(st, n, g, rs);
        } else {
            k_pauli_diag<T, false><<<grid, kReduceThreads, 0, s>>>(st, n, g, rs);
        }
    } else {
        k_pauli_group<T><<<kReduceBlocks, kReduceThreads, 0, s>>>((const cx<T> *)st, n, g, rs);
    }
    count_launch();
    return cudaGetLastError();
}

// ---- tiled pass over many pair-form strings ---------------------------------------
// One tile of 2^K amplitudes (32 KiB, TMA) per CTA iteration, three CTAs per SM
// that overlap one's load with the others' sums.  (Two buffers per CTA leave
// the running sums too little L1: 5.7 -> 6.6 ms on the case below.)  An
// amplitude's (re, im) is one packed operand: a pair's product is an f32x2
// multiplication whose lanes (re re and im im, or re im and im re) are summed
// apart until the end, so 12 packed instructions form and add one pair.
// A product is its rounded high part plus the exact error and the cross terms
// (complex128: the tile holds float-float amplitudes, binary64 split once per
// tile); it is added without normalising (PauliSum).
// Strings whose flips lie within three neighbouring tile bits run in windows:
// a thread holds the 8 amplitudes of its window in registers, read once for
// all strings of the window, and a pair is two registers.  Lane l takes the
// amplitudes in the order j ^ (l >> w) below bit 3, so the reads spread over
// the banks; the flip mask still pairs j with j ^ x.  Other strings read both
// amplitudes of every pair.  Strings with one flip mask and part (Re or Im)
// form a group: the products are formed once and every string adds them with
// its signs.
// Tile sums gather in three floats and go to binary64 every kPauliFlush tiles:
// a conversion per string and tile kept GB300's FP64 pipe busy half of the
// time.
// Measured, the 27 X strings of a ring TFIM on 27 qubits in float-float, four
// passes: 5.8 -> 4.2 ms (a pass that only reads: 0.38 ms).  With sums of two
// floats it was 4.0 ms, and a string's value less exact than before (14
// qubits, random states, rms: binary64 sums per tile 4.2e-17, two floats
// 5.4e-17, three 2.5e-17; complex64 1.8e-17, 2.6e-17, 1.0e-17).
__device__ __forceinline__ uint64_t tile_base_of(uint64_t tau, uint32_t l, uint32_t m, const uint8_t *hq) {
    uint64_t b = tau << l;
    for (uint32_t j = 0; j < m; j++) b = insert_zero(b, hq[j]);
    return b;
}

constexpr int kPauliThreads = kReduceThreads, kPauliFlush = 32;

__device__ __forceinline__ float2 flip_signs(float2 v, uint32_t s) {
    return make_float2(__uint_as_float(__float_as_uint(v.x) ^ s), __uint_as_float(__float_as_uint(v.y) ^ s));
}
template <bool FFV>
__device__ __forceinline__ ff2::v2 pauli_amp(const void *tile, uint32_t u) {
    ff2::v2 a{};
    if constexpr (FFV) a = reinterpret_cast<const ff2::v2 *>(tile)[u];
    else a.h = reinterpret_cast<const float2 *>(tile)[u];
    return a;
}
// conj(a) b as h + l, lane by lane: Re = re re + im im, Im = re im - im re (the
// lanes' difference; one scalar instruction per lane, no exchanged operands)
template <bool FFV, bool IM>
__device__ __forceinline__ ff2::v2 pauli_product(const ff2::v2 &a, const ff2::v2 &b) {
    if constexpr (IM) {
        const float2 p = make_float2(__fmul_rn(a.h.x, b.h.y), __fmul_rn(a.h.y, b.h.x));
        float2 lo = make_float2(__fmaf_rn(a.h.x, b.h.y, -p.x), __fmaf_rn(a.h.y, b.h.x, -p.y));
        if constexpr (FFV) {
            lo = make_float2(__fmaf_rn(a.h.x, b.l.y, lo.x), __fmaf_rn(a.h.y, b.l.x, lo.y));
            lo = make_float2(__fmaf_rn(a.l.x, b.h.y, lo.x), __fmaf_rn(a.l.y, b.h.x, lo.y));
        }
        return ff2::v2{p, lo};
    }
    const float2 p = ff2::mul(a.h, b.h);
    float2 lo = ff2::fma(a.h, b.h, flip_signs(p, 0x80000000u));
    if constexpr (FFV) lo = ff2::fma(a.l, b.h, ff2::fma(a.h, b.l, lo));
    return ff2::v2{p, lo};
}
// A sum over a tile, lane by lane: the products' high parts, their low parts
// and the errors of adding the high ones, each in a sum of its own (joined
// after every product they round where the start of this chain is longest:
// rms error of a thread's sum 2.4e-15 -> 1.1e-15 of itself in complex64,
// 3.7e-15 -> 2.7e-15 in float-float, at the same number of instructions).
struct PauliSum {
    float2 h, lo, er;
};
__device__ __forceinline__ void pauli_add(PauliSum &S, float2 p, float2 lo) {
    const ff2::v2 t = ff2::two_sum(S.h, p);
    S = PauliSum{t.h, ff2::add(S.lo, lo), ff2::add(S.er, t.l)};
}
// a thread's sum over the tile, its lanes joined, into the string's running
// sum.  Float-float states keep the running sum's rounding errors too: the
// sums of complex64 products have the bits to spare (32 tiles: 0.8e-14 of one
// tile's sum; in plain float-float 2.5e-14).
template <bool FFV, bool IM>
__device__ __forceinline__ void pauli_tail(const PauliSum &S, bool neg, f3 &acc) {
    const float sn = neg ? -1.f : 1.f, sy = IM ? -sn : sn;
    const ff::f2 t = ff::two_sum(__fmul_rn(S.h.x, sn), __fmul_rn(S.h.y, sy)), r = ff::two_sum(acc.h, t.h);
    const float lo = __fmaf_rn(S.lo.x, sn, __fmul_rn(S.lo.y, sy));
    const float er = ff::add(__fmaf_rn(S.er.x, sn, __fmaf_rn(S.er.y, sy, t.l)), r.l);
    if constexpr (FFV) {
        const ff::f2 g = ff::two_sum(acc.m, lo), k = ff::two_sum(g.h, er);
        acc = f3{r.h, k.h, ff::add(acc.l, ff::add(g.l, k.l))};
    } else {
        acc = f3{r.h, ff::add(acc.m, lo), ff::add(acc.l, er)};
    }
}

// The strings of one window with flip mask X and part IM: the four products,
// then every string's signed sum.
template <bool FFV, bool IM, int X>
__device__ __forceinline__ void window_group(const PauliTilePass &p, const ff2::v2 (&a)[8], uint32_t &k, uint32_t w,
                                             uint32_t F, uint32_t negs, uint32_t signs, f3 *acc) {
    constexpr int hb = X >= 4 ? 2 : (X >= 2 ? 1 : 0);
    ff2::v2 c[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int j = ((i >> hb) << (hb + 1)) | (i & ((1 << hb) - 1));
        c[i] = pauli_product<FFV, IM>(a[j], a[j ^ X]);
    }
    const uint32_t end = p.t[k].group_end;
#pragma unroll 1
    for (; k < end; k++) {
        PauliSum S{c[0].h, c[0].l, make_float2(0.f, 0.f)};
        bool neg = ((negs >> k) & 1u) != 0;
        if ((signs >> k) & 1u) {
            const uint32_t zl = p.t[k].zl, zr = zl >> w;
            neg ^= (__popc(F & zl) & 1) != 0;
#pragma unroll
            for (int i = 1; i < 4; i++) {  // (j = 0 has no sign of its own)
                const uint32_t j = ((i >> hb) << (hb + 1)) | (i & ((1 << hb) - 1));
                const uint32_t sg = (uint32_t)__popc(j & zr) << 31;
                pauli_add(S, flip_signs(c[i].h, sg), flip_signs(c[i].l, sg));
            }
        } else {
#pragma unroll
            for (int i = 1; i < 4; i++) pauli_add(S, c[i].h, c[i].l);
        }
        pauli_tail<FFV, IM>(S, neg, acc[k]);
    }
}

// Every string of one window, terms from k0.  Bit k of negs: the parity of
// string k's phase mask on the tile's base; of signs: string k has phases
// inside the tile.
template <bool FFV>
__device__ __forceinline__ void pauli_window(const PauliTilePass &p, const void *tile, uint32_t k0, uint32_t negs,
                                             uint32_t signs, f3 *acc) {
    const uint32_t w = p.t[k0].w, low = (1u << w) - 1u, groups = p.t[k0].groups;
    for (uint32_t q = threadIdx.x; q < (1u << (p.K - 3)); q += kPauliThreads) {
        const uint32_t sw = w < 3 ? ((threadIdx.x & 31u) >> w) & 7u : 0u;
        const uint32_t F = (q & low) | ((q & ~low) << 3) | (sw << w);
        ff2::v2 a[8];
#pragma unroll
        for (int j = 0; j < 8; j++) a[j] = pauli_amp<FFV>(tile, F ^ ((uint32_t)j << w));
        uint32_t k = k0;
#define KBWG_WX(X)                                                                                    \
    if (groups & (1u << (2 * X))) window_group<FFV, false, X>(p, a, k, w, F, negs, signs, acc); \
    if (groups & (2u << (2 * X))) window_group<FFV, true, X>(p, a, k, w, F, negs, signs, acc);
        KBWG_WX(1) KBWG_WX(2) KBWG_WX(3) KBWG_WX(4) KBWG_WX(5) KBWG_WX(6) KBWG_WX(7)
#undef KBWG_WX
    }
}

// C strings k0.. of one group over the tile, both amplitudes of a pair read.
template <bool FFV, bool IM, int C>
__device__ __forceinline__ void pauli_group_terms(const PauliTilePass &p, const void *tile, uint32_t k0, uint32_t negs,
                                                  f3 *acc) {
    const uint32_t xl = p.t[k0].xl, pairs = 1u << (p.K - 1);
    const uint32_t keep = (1u << p.t[k0].hb) - 1u;
    PauliSum S[C];
    uint32_t zl[C];
#pragma unroll
    for (int c = 0; c < C; c++) {
        S[c] = PauliSum{make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        zl[c] = p.t[k0 + c].zl;
    }
#pragma unroll 4
    for (uint32_t q = threadIdx.x; q < pairs; q += kPauliThreads) {
        const uint32_t u = q + (q & ~keep);  // the highest flipped bit clear
        const ff2::v2 w = pauli_product<FFV, IM>(pauli_amp<FFV>(tile, u), pauli_amp<FFV>(tile, u ^ xl));
#pragma unroll
        for (int c = 0; c < C; c++) {
            const uint32_t sg = (uint32_t)__popc(u & zl[c]) << 31;
            pauli_add(S[c], flip_signs(w.h, sg), flip_signs(w.l, sg));
        }
    }
#pragma unroll
    for (int c = 0; c < C; c++) pauli_tail<FFV, IM>(S[c], ((negs >> (k0 + c)) & 1u) != 0, acc[k0 + c]);
}

template <bool FFV, bool IM>
__device__ __forceinline__ void pauli_group(const PauliTilePass &p, const void *tile, uint32_t k0, uint32_t k1,
                                            uint32_t negs, f3 *acc) {
    for (; k0 + 2 <= k1; k0 += 2) pauli_group_terms<FFV, IM, 2>(p, tile, k0, negs, acc);
    if (k0 < k1) pauli_group_terms<FFV, IM, 1>(p, tile, k0, negs, acc);
}

template <class T, bool kFF>
__global__ void __launch_bounds__(kPauliThreads, 3) k_pauli_tile(const void *__restrict__ st, uint32_t n,
                                                                 const __grid_constant__ PauliTilePass p,
                                                                 ReduceScratch rs, int *err) {
    constexpr bool FFV = sizeof(T) == 8;
    constexpr uint32_t kElem = FFV ? 16 : 8;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const uint32_t K = p.K, l = p.l, m = p.m, nt = p.nterms;
    const uint32_t N = 1u << K, tile_bytes = kElem << K;
    uint64_t *chunk_off = reinterpret_cast<uint64_t *>(smem_raw + tile_bytes);
    uint64_t *bar = chunk_off + (1u << m);
    for (uint32_t c = threadIdx.x; c < (1u << m); c += blockDim.x) {
        uint64_t off = 0;
        for (uint32_t j = 0; j < m; j++) off |= (uint64_t)((c >> j) & 1u) << p.hq[j];
        chunk_off[c] = off;
    }
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        fence_mbar_init();
    }
    const uint64_t tiles = 1ull << (n - K);
    f3 acc[kMaxTerms];  // (local memory, touched once per string and tile)
    double wide[kMaxTerms];
    bool flushed = false;
    for (int k = 0; k < kMaxTerms; k++) acc[k] = f3{0.f, 0.f, 0.f};
    __syncthreads();
    auto issue_load = [&](uint64_t tau) {
        if (threadIdx.x < 32) {
            const uint64_t base = tile_base_of(tau, l, m, p.hq);
            if (threadIdx.x == 0) mbar_expect_tx(bar, tile_bytes);
            __syncwarp();
            for (uint32_t c = threadIdx.x; c < (1u << m); c += 32)
                tma_load(smem_raw + ((size_t)(c << l) * kElem), (const char *)st + (base + chunk_off[c]) * kElem,
                         kElem << l, bar);
        }
    };
    if (blockIdx.x < tiles) issue_load(blockIdx.x);
    // lane k keeps string k's phase mask outside the tile
    const uint32_t my = threadIdx.x & 31u;
    const uint64_t my_zo = my < nt ? p.t[my].zo : 0ull;
    const uint32_t signs = __ballot_sync(0xffffffffu, my < nt && p.t[my].zl != 0u);
    uint32_t it = 0;
    for (uint64_t tau = blockIdx.x; tau < tiles; tau += gridDim.x, it++) {
        const uint64_t base = tile_base_of(tau, l, m, p.hq);
        void *tile = smem_raw;
        const uint32_t negs = __ballot_sync(0xffffffffu, (__popcll(base & my_zo) & 1) != 0);
        if (!tile_wait(bar, it & 1u, err)) break;  // (the sums are not valid; the ticket still counts)
        if constexpr (FFV && !kFF) {
            for (uint32_t u = threadIdx.x; u < N; u += kPauliThreads) {
                const cx<double> a = reinterpret_cast<const cx<double> *>(tile)[u];
                // (rounded, not cut: the low parts half as large and of both signs)
                ff::f2 r = ff::from_double(a.re), i = ff::from_double(a.im);
                r = ff::fast_two_sum(r.h, r.l);
                i = ff::fast_two_sum(i.h, i.l);
                reinterpret_cast<ff2::v2 *>(tile)[u] = ff2::v2{make_float2(r.h, i.h), make_float2(r.l, i.l)};
            }
            __syncthreads();
        }
#pragma unroll 1
        for (uint32_t k0 = 0; k0 < nt;) {
            if (p.t[k0].w < 32u) {
                pauli_window<FFV>(p, tile, k0, negs, signs, acc);
                k0 = p.t[k0].window_end;
            } else {
                const uint32_t k1 = p.t[k0].group_end;
                if (p.t[k0].im) pauli_group<FFV, true>(p, tile, k0, k1, negs, acc);
                else pauli_group<FFV, false>(p, tile, k0, k1, negs, acc);
                k0 = k1;
            }
        }
        fence_proxy_async();
        __syncthreads();
        if (tau + gridDim.x < tiles) issue_load(tau + gridDim.x);
        if ((it + 1) % (uint32_t)kPauliFlush == 0) {
            for (int k = 0; k < (int)nt; k++) {
                wide[k] = (flushed ? wide[k] : 0.0) + to_double(acc[k]);
                acc[k] = f3{0.f, 0.f, 0.f};
            }
            flushed = true;
        }
    }
    const int lane = threadIdx.x & 31;
    double mine = 0.0;
    if (flushed)  // (uniform over the block)
        for (int k = 0; k < (int)nt; k++) {
            const double v = warp_sum(wide[k]);
            if (lane == k) mine = v;
        }
    mine += to_double(warp_sum_terms([&](int k) {
        const ff::f2 t = ff::two_sum(acc[k].m, acc[k].l);
        return f3{acc[k].h, t.h, t.l};
    }));
    finish_terms(lane < (int)nt ? mine * p.t[lane].factor : 0.0, nt, rs);
}

template <class T>
cudaError_t launch_pauli_tile(const void *st, uint32_t n, bool ff_resident, const PauliTilePass &p,
                              const ReduceScratch &rs, int *err, cudaStream_t s) {
    auto bytes = [](uint32_t K, uint32_t m) -> size_t {
        return ((size_t)(sizeof(T) == 8 ? 16 : 8) << K) + (sizeof(uint64_t) << m) + 16;
    };
    auto kern = (sizeof(T) == 8 && ff_resident) ? k_pauli_tile<T, true> : k_pauli_tile<T, false>;
    constexpr uint32_t kMax = pauli_tile_bits<T>();  // (the limit is set once per kernel, for its largest tile)
    cudaError_t e = ensure_smem_limit((const void *)kern, bytes(kMax, kMax - 5));
    if (e != cudaSuccess) return e;
    const uint64_t tiles = 1ull << (n - p.K);
    const unsigned grid = (unsigned)std::min<uint64_t>(tiles, 152ull * 3);
    kern<<<grid, kPauliThreads, bytes(p.K, p.m), s>>>(st, n, p, rs, err);
    count_launch();
    return cudaGetLastError();
}

// ---- support test for dump / sample ---------------------------------------
// Reference: hypot(re, im) > F(eps) in F (src/dense.rs:374).  With hypot
// correctly rounded this is re^2 + im^2 > m^2, m the midpoint between F(eps)
// and the next F value; decided in double with a guard band, and with an
// exact double evaluation inside the band.
__device__ __forceinline__ bool above_eps(cx<float> a) {
    const float q = __fmaf_rn(a.re, a.re, __fmul_rn(a.im, a.im));
    const float lo = 9.99998e-13f, hi = 1.000002e-12f;  // band around (1e-6)^2
    if (q > hi) return true;
    if (q < lo) return false;
    const double e = (double)1e-6f, e_next = (double)__int_as_float(__float_as_int(1e-6f) + 1);
    const double mid = 0.5 * (e + e_next);
    const double x = (double)a.re * (double)a.re + (double)a.im * (double)a.im;
    return x > mid * mid;
}
__device__ __forceinline__ bool above_eps(cx<double> a) {
    const double q = a.re * a.re + a.im * a.im;
    return q > 1e-30;
}

template <class T>
__device__ __forceinline__ double weight(cx<T> a) {
    if (!above_eps(a)) return 0.0;
    const double r = (double)a.re, i = (double)a.im;
    return __fma_rn(r, r, __dmul_rn(i, i));
}

// Weight of amplitude i of a state of either type or form, in binary64: a
// float-float amplitude is what ensure_binary64 would make of it.
template <class T, bool kFF>
__device__ __forceinline__ double weight_at(const void *st, uint64_t i) {
    if constexpr (kFF) {
        const float4 f = reinterpret_cast<const float4 *>(st)[i];  // re.hi, im.hi, re.lo, im.lo
        return weight(cx<double>{ff::to_double(ff::f2{f.x, f.z}), ff::to_double(ff::f2{f.y, f.w})});
    } else {
        return weight(reinterpret_cast<const cx<T> *>(st)[i]);
    }
}

int dump_blocks(uint32_t n) {
    const uint64_t ns = 1ull << n;
    uint64_t R = ns / 4096;
    if (R < 256) R = 256;
    if (R > ns) R = ns;
    return (int)(ns / R);
}
int sample_blocks(uint32_t n) { return dump_blocks(n); }

template <class T>
__global__ void __launch_bounds__(256) k_dump_count(const cx<T> *__restrict__ st, uint64_t R, uint64_t *counts) {
    const uint64_t base = (uint64_t)blockIdx.x * R;
    unsigned c = 0;
    for (uint64_t i = threadIdx.x; i < R; i += blockDim.x) c += above_eps(st[base + i]) ? 1u : 0u;
    const double t = block_sum((double)c);
    if (threadIdx.x == 0) counts[blockIdx.x] = (uint64_t)t;
}

template <class T>
__global__ void __launch_bounds__(256)
    k_dump_write(const cx<T> *__restrict__ st, uint64_t R, const uint64_t *offsets, DumpSpec spec, uint64_t *states,
                 double *re, double *im) {
    __shared__ unsigned wcount[8];
    __shared__ uint8_t q[64];
    if (threadIdx.x < 64) q[threadIdx.x] = spec.qubits[threadIdx.x];
    const uint64_t base = (uint64_t)blockIdx.x * R;
    uint64_t running = offsets[blockIdx.x];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    for (uint64_t c0 = 0; c0 < R; c0 += blockDim.x) {
        const uint64_t i = c0 + threadIdx.x;
        bool keep = false;
        cx<T> a{};
        if (i < R) {
            a = st[base + i];
            keep = above_eps(a);
        }
        const unsigned bal = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) wcount[w] = __popc(bal);
        __syncthreads();
        unsigned before = 0, total = 0;
        for (int k = 0; k < (int)(blockDim.x >> 5); k++) {
            if (k < w) before += wcount[k];
            total += wcount[k];
        }
        if (keep) {
            const uint64_t pos = running + before + __popc(bal & ((1u << lane) - 1));
            const uint64_t s = base + i;
            uint64_t packed = 0;
            for (uint32_t j = 0; j < spec.nq; j++) packed |= ((s >> q[spec.nq - 1 - j]) & 1ull) << j;
            states[pos] = packed;
            re[pos] = (double)a.re;
            im[pos] = (double)a.im;
        }
        running += total;
        __syncthreads();
    }
}

template <class T>
cudaError_t launch_dump_count(const void *st, uint32_t n, uint64_t *counts, cudaStream_t s) {
    const int B = dump_blocks(n);
    const uint64_t R = (1ull << n) / B;
    k_dump_count<T><<<B, 256, 0, s>>>((const cx<T> *)st, R, counts);
    count_launch();
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_dump_write(const void *st, uint32_t n, const uint64_t *offsets, const DumpSpec &spec,
                              uint64_t *states, double *re, double *im, cudaStream_t s) {
    const int B = dump_blocks(n);
    const uint64_t R = (1ull << n) / B;
    k_dump_write<T><<<B, 256, 0, s>>>((const cx<T> *)st, R, offsets, spec, states, re, im);
    count_launch();
    return cudaGetLastError();
}

// ---- sampling -------------------------------------------------------------------
// The block sums only say which block a shot falls into; the picks scan the few
// blocks that hold one.  (Scanning every block here too kept the FP64 pipe busy
// for 372 us on 24 qubits.)  The scan's total may differ from the sum in the
// last bits: a shot between the two takes the block's last amplitude with a
// weight.  The sums are no less exact than in binary64, which float-float ones
// are not (they move the border between two blocks by up to 2^-49 of it):
// complex64 and binary64 states on the FP64 pipe, float-float states as three
// floats per part, whose roundings stay below 2^-60 (24 qubits, a whole
// experiment: on the FP64 pipe, after ensure_binary64's conversion of every
// amplitude, 0.39 ms more).
template <class T, bool kFF>
__global__ void __launch_bounds__(256) k_weight_blocksum(const void *__restrict__ st, uint64_t R, double *blocksum) {
    const uint64_t base = (uint64_t)blockIdx.x * R;
    double sum = 0.0;
    if constexpr (!kFF) {
#pragma unroll 4
        for (uint64_t i = threadIdx.x; i < R; i += 256) sum += weight_at<T, kFF>(st, base + i);
    } else {
        const float4 *amp = reinterpret_cast<const float4 *>(st) + base;  // re.hi, im.hi, re.lo, im.lo
        float2 ah = make_float2(0.f, 0.f), am = ah, al = ah;
#pragma unroll 4
        for (uint64_t i = threadIdx.x; i < R; i += 256) {
            const float4 f = amp[i];
            float2 h = make_float2(f.x, f.y), l = make_float2(f.z, f.w);
            float2 p = ff2::mul(h, h);
            const float q = __fadd_rn(p.x, p.y);
            if (!(q > 1.00001e-30f) && !(q > 0.99999e-30f && weight_at<T, true>(st, base + i) > 0.0))
                h = l = p = make_float2(0.f, 0.f);  // (no weight: see weight())
            const float2 e = ff2::fma(h, h, ff2::neg(p)), l2 = ff2::add(l, l), c = ff2::mul(h, l2);
            const float2 ec = ff2::fma(h, l2, ff2::neg(c));  // p + e + c + ec + l l: the squares
            const ff2::v2 t = ff2::two_sum(ah, p), u = ff2::two_sum(am, t.l), v = ff2::two_sum(u.h, e),
                          w = ff2::two_sum(v.h, c);
            ah = t.h;
            am = w.h;
            al = ff2::add(al, ff2::fma(l, l, ff2::add(ff2::add(u.l, v.l), ff2::add(w.l, ec))));
        }
        sum = to_double(add(f3{ah.x, am.x, al.x}, f3{ah.y, am.y, al.y}));
    }
    const double t = block_sum(sum);
    if (threadIdx.x == 0) blocksum[blockIdx.x] = t;
}

template <class T, bool kFF>
__global__ void __launch_bounds__(256)
    k_sample_pick(const void *__restrict__ st, uint64_t R, const uint32_t *blocks, const uint64_t *shot_begin,
                  const double *prefix, const double *chosen, uint64_t *pick) {
    __shared__ double pre[256];
    __shared__ uint64_t last_nz;
    const uint32_t b = blocks[blockIdx.x];
    const uint64_t base = (uint64_t)b * R;
    const double P = prefix[blockIdx.x];
    uint64_t sh = shot_begin[blockIdx.x];
    const uint64_t sh_end = shot_begin[blockIdx.x + 1];
    double running = 0.0;
    if (threadIdx.x == 0) last_nz = base;
    __syncthreads();
    for (uint64_t c0 = 0; c0 < R && sh < sh_end; c0 += blockDim.x) {
        const uint64_t i = c0 + threadIdx.x;
        const double w = (i < R) ? weight_at<T, kFF>(st, base + i) : 0.0;
        double total;
        const double incl = block_inclusive_scan(w, &total);
        pre[threadIdx.x] = P + (running + incl);
        if (w > 0.0) atomicMax((unsigned long long *)&last_nz, (unsigned long long)(base + i));
        __syncthreads();
        const double chunk_end = pre[blockDim.x - 1];
        // shots whose first prefix above `chosen` lies in this chunk
        while (sh < sh_end && chosen[sh] < chunk_end) {
            const uint64_t j = sh + threadIdx.x;
            const bool here = j < sh_end && chosen[j] < chunk_end;
            if (here) {
                const double c = chosen[j];
                int lo = 0, hi = blockDim.x - 1;  // first pre[] > c
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (pre[mid] > c)
                        hi = mid;
                    else
                        lo = mid + 1;
                }
                pick[j] = base + c0 + lo;
            }
            // past every shot resolved in this chunk (they are sorted, so those
            // here come first; counting them one by one in every thread took
            // 80 of the 87 us of 1024 shots on one state of 2^12)
            sh += (uint64_t)__syncthreads_count(here);
        }
        running = running + total;
        __syncthreads();
    }
    // rounding leftovers: the block's last element with weight
    for (uint64_t j = sh + threadIdx.x; j < sh_end; j += blockDim.x) pick[j] = last_nz;
}

template <class T>
cudaError_t launch_weight_blocksum(const void *st, uint32_t n, bool ff_resident, double *blocksum, cudaStream_t s) {
    const int B = sample_blocks(n);
    const uint64_t R = (1ull << n) / B;
    if (sizeof(T) == 8 && ff_resident) k_weight_blocksum<double, true><<<B, 256, 0, s>>>(st, R, blocksum);
    else k_weight_blocksum<T, false><<<B, 256, 0, s>>>(st, R, blocksum);
    count_launch();
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_sample_pick(const void *st, uint32_t n, bool ff_resident, const uint32_t *blocks,
                               uint32_t nblocks_with_shots,
                               const uint64_t *shot_begin, const double *prefix, const double *chosen,
                               uint64_t *pick, cudaStream_t s) {
    const int B = sample_blocks(n);
    const uint64_t R = (1ull << n) / B;
    if (nblocks_with_shots == 0) return cudaSuccess;
    if (sizeof(T) == 8 && ff_resident)
        k_sample_pick<double, true><<<nblocks_with_shots, 256, 0, s>>>(st, R, blocks, shot_begin, prefix, chosen, pick);
    else
        k_sample_pick<T, false><<<nblocks_with_shots, 256, 0, s>>>(st, R, blocks, shot_begin, prefix, chosen, pick);
    count_launch();
    return cudaGetLastError();
}

// ---- allocation-free masked norm ----------------------------------------------
// Some callers of this library cannot allocate device memory: code that runs
// while a CUDA graph is being captured (cudaMalloc is not capturable), plugins
// hosted by a runtime that owns every device allocation through its own pool,
// and real-time loops that cannot take the implicit synchronisation of an
// allocation.  kbwg_masked_norm_noalloc serves them: it runs the same
// reduction as kbwg_measure_p1 but keeps its scratch (608 per-block partial
// sums and the last-block ticket) in the fixed device array below instead of
// a per-handle cudaMalloc.  Every GPU that loads this library holds the array
// (8 KiB) until the process exits.
constexpr size_t kNoAllocScratchBytes = 8192;
constexpr size_t kNoAllocTicketOffset = 4864;  // after kReduceBlocks doubles, 256-aligned
static_assert(kReduceBlocks * sizeof(double) <= kNoAllocTicketOffset, "partials overflow the fixed scratch");
static_assert(kNoAllocTicketOffset + 256 <= kNoAllocScratchBytes, "ticket overflows the fixed scratch");
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

// Host code may not use g_noalloc_scratch as an address (it names a host-side
// stand-in); the device address is looked up with the device current, once
// per CUDA context.  The cache is keyed on the context's id, not on the
// device ordinal: after cudaDeviceReset the device gets a new context in
// which the array may have another address.
namespace {
typedef int (*CtxGetCurrentFn)(void **);
typedef int (*CtxGetIdFn)(void *, unsigned long long *);
std::mutex g_noalloc_mu;
std::vector<std::pair<unsigned long long, void *>> g_noalloc_addr;  // context id -> array address

// Id of the calling thread's current CUDA context (driver entry points
// obtained through the runtime); false if none is current or unknown.
bool current_context_id(unsigned long long &id) {
    static CtxGetCurrentFn get_current = nullptr;
    static CtxGetIdFn get_id = nullptr;
    static bool resolved = false;
    if (!resolved) {
        resolved = true;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", (void **)&get_current, 12000, cudaEnableDefault,
                                             &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
            get_current = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", (void **)&get_id, 12000, cudaEnableDefault, &q) !=
                cudaSuccess || q != cudaDriverEntryPointSuccess)
            get_id = nullptr;
    }
    void *ctx = nullptr;
    if (!get_current || !get_id || get_current(&ctx) != 0 || !ctx) return false;
    return get_id(ctx, &id) == 0;
}
}  // namespace

static cudaError_t noalloc_scratch(void **out) {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    unsigned long long id = 0;
    if (current_context_id(id))
        for (const auto &a : g_noalloc_addr)
            if (a.first == id) {
                *out = a.second;
                return cudaSuccess;
            }
    // set-up on this context (the lookup makes the current device's context current if none is)
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return e;
    if (current_context_id(id)) g_noalloc_addr.emplace_back(id, p);
    *out = p;
    return cudaSuccess;
}

// A device or managed allocation on the current device (a host pointer, or
// memory of another device, would make the kernel fault).
static bool on_current_device(const void *p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (a.type != cudaMemoryTypeDevice && a.type != cudaMemoryTypeManaged) return false;
    int dev = -1;
    return cudaGetDevice(&dev) == cudaSuccess && a.device == dev;
}

}  // namespace kbwg

extern "C" int32_t kbwg_masked_norm_noalloc(const void *state, uintptr_t num_qubits, int32_t precision,
                                            uint64_t mask, uint64_t value, double *out, void *stream) {
    using namespace kbwg;
    if (!state || !out) {
        set_error(KBWG_EINVAL, "kbwg_masked_norm_noalloc: null state or output pointer");
        return KBWG_EINVAL;
    }
    if (num_qubits > 32) {
        set_error(KBWG_EQUBITS, "kbwg_masked_norm_noalloc: at most 32 qubits (its fixed scratch serves "
                                "a 608-block grid over up to 2^32 amplitudes)");
        return KBWG_EQUBITS;
    }
    if (precision != KBWG_C64 && precision != KBWG_C128) {
        set_error(KBWG_EINVAL, "kbwg_masked_norm_noalloc: bad precision");
        return KBWG_EINVAL;
    }
    const uint64_t all = (1ull << num_qubits) - 1;  // num_qubits <= 32 here
    if ((mask & ~all) || (value & ~mask)) {
        set_error(KBWG_EINVAL, "kbwg_masked_norm_noalloc: mask/value outside the register or value outside mask");
        return KBWG_EINVAL;
    }
    if (!on_current_device(state) || !on_current_device(out)) {
        set_error(KBWG_EINVAL, "kbwg_masked_norm_noalloc: state and out must be device (or managed) memory of the "
                               "current device");
        return KBWG_EINVAL;
    }
    void *base = nullptr;
    cudaError_t e = noalloc_scratch(&base);
    if (e != cudaSuccess) {
        set_error(KBWG_ECUDA, std::string("kbwg_masked_norm_noalloc: scratch lookup: ") + cudaGetErrorString(e));
        return KBWG_ECUDA;
    }
    ReduceScratch rs;
    rs.partials = (double *)base;
    rs.ticket = (unsigned *)((char *)base + kNoAllocTicketOffset);
    rs.result = out;
    cudaStream_t s = (cudaStream_t)stream;
    e = cudaMemsetAsync(rs.ticket, 0, sizeof(unsigned), s);  // the array keeps the last call's contents
    if (e == cudaSuccess)
        e = precision ? launch_masked_norm<double>(state, (uint32_t)num_qubits, mask, value, rs, s)
                      : launch_masked_norm<float>(state, (uint32_t)num_qubits, mask, value, rs, s);
    if (e != cudaSuccess) {
        set_error(KBWG_ECUDA, std::string("kbwg_masked_norm_noalloc: ") + cudaGetErrorString(e));
        return KBWG_ECUDA;
    }
    return KBWG_OK;
}

namespace kbwg {

#define INST(T)                                                                                               \
    template cudaError_t launch_masked_norm<T>(const void *, uint32_t, uint64_t, uint64_t, const ReduceScratch &, \
                                               cudaStream_t);                                                 \
    template cudaError_t launch_measure_steps<T>(const void *, uint32_t, MeasureCtl *, uint32_t,               \
                                                 const ReduceScratch &, cudaStream_t);                        \
    template cudaError_t launch_collapse<T>(void *, uint32_t, const MeasureCtl *, uint64_t, uint64_t, double,   \
                                            cudaStream_t);                                                    \
    template cudaError_t launch_pauli_group<T>(const void *, uint32_t, const PauliGroup &, const ReduceScratch &, \
                                               cudaStream_t, bool);                                           \
    template cudaError_t launch_pauli_small<T>(const void *, uint32_t, const PauliSmall &, const ReduceScratch &, \
                                               cudaStream_t);                                                 \
    template cudaError_t launch_pauli_tile<T>(const void *, uint32_t, bool, const PauliTilePass &,               \
                                              const ReduceScratch &, int *, cudaStream_t);                           \
    template cudaError_t launch_dump_count<T>(const void *, uint32_t, uint64_t *, cudaStream_t);               \
    template cudaError_t launch_dump_write<T>(const void *, uint32_t, const uint64_t *, const DumpSpec &,        \
                                              uint64_t *, double *, double *, cudaStream_t);                  \
    template cudaError_t launch_weight_blocksum<T>(const void *, uint32_t, bool, double *, cudaStream_t);      \
    template cudaError_t launch_sample_pick<T>(const void *, uint32_t, bool, const uint32_t *, uint32_t,       \
                                               const uint64_t *, const double *, const double *, uint64_t *,  \
                                               cudaStream_t);
INST(float)
INST(double)

}  // namespace kbwg

// BatchNorm forward / backward for [b, z, rc] fp32 tensors (NCHW with rc = H*W).
// Replaces gpu_batchnorm_forward_{1,2,3} / gpu_batchnorm_backward_{1,2,3}
// (EDDL src/hardware/gpu/nn/gpu_bn_kernels.cu:92-204, host gpu_bn.cu:65-117); the
// arithmetic follows cpu_batchnorm_forward / cpu_batchnorm_backward
// (src/hardware/cpu/nn/cpu_bn.cpp:118-249) operation by operation.
//
// One launch per direction for small tensors (bn_*_one_kernel: a channel is kept in shared
// memory and read once), otherwise two, each a single streaming pass:
//   stats : grid (z, S)  every block reduces one slice of one channel with float4
//           loads and warp shuffles and stores a partial (sum, sumsq) pair;
//   apply : grid (z, S)  every block re-reduces its channel's S partials in double
//           (deterministic, no atomics), derives the per-channel constants and
//           streams its slice: normalise (+affine, + optional fused ReLU output) or
//           the backward formula.  Block y == 0 also writes the per-channel outputs.
// Traffic per element: forward 12 bytes (x, opa, y; +4 where the ReLU of y is written too),
// backward 16 (delta, opa; delta *= gamma in place as in the reference, parent delta);
// two-pass +4 and +8.
#include <cooperative_groups.h>
#include <atomic>
#include <mutex>
#include "common.cuh"

namespace {

using namespace eb;

constexpr int kBlock = 256;
constexpr int kMaxSplit = 256;

struct Slice { unsigned begin, end; };   // element range inside one channel's b*rc items

__device__ __forceinline__ Slice slice_of(unsigned per_channel, unsigned nsplit, unsigned s) {
    // chunk is a multiple of 4 so float4 accesses never straddle slices
    unsigned chunk = ((per_channel + nsplit - 1) / nsplit + 3u) & ~3u;
    Slice r;
    r.begin = min(s * chunk, per_channel);
    r.end = min(r.begin + chunk, per_channel);
    return r;
}

// Quotients by one divisor.  The reference divides every element by its channel's sigma, and an IEEE division per element is a third
// of a BatchNorm kernel's instructions.  With the correctly rounded reciprocal r of the divisor in hand, Markstein's method (P. Markstein, Computation of elementary functions on
// the IBM RISC System/6000 processor, 1990) gives the same correctly rounded quotient in five multiply-adds: q = a r, one
// correction makes q faithful, a second one with the exact remainder rounds it correctly.  It needs every intermediate in
// the normal range: dividends outside 2^-60 .. 2^60 (zeros, infinities and NaNs among them) and divisors outside 2^-30 .. 2^30 take
// the ordinary division.
struct Divisor {
    float b, r; bool plain;
    __device__ __forceinline__ float fast(float a) const {
        float q = __fmul_rn(a, r);
        q = __fmaf_rn(__fmaf_rn(-q, b, a), r, q);
        return __fmaf_rn(__fmaf_rn(-q, b, a), r, q);
    }
    __device__ __forceinline__ float operator()(float a) const {
        const float m = fabsf(a);
        return !plain && m > 8.6736174e-19f && m < 1.1529215e18f ? fast(a) : __fdiv_rn(a, b);
    }
    __device__ __forceinline__ float4 operator()(float4 a) const {
        const float lo = fminf(fminf(fabsf(a.x), fabsf(a.y)), fminf(fabsf(a.z), fabsf(a.w)));
        const float hi = fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(a.w)));
        // a NaN among the four passes neither fminf nor fmaxf: the sum keeps it
        const float sum = (a.x + a.y) + (a.z + a.w);
        if (!plain && lo > 8.6736174e-19f && hi < 1.1529215e18f && sum == sum) return make_float4(fast(a.x), fast(a.y), fast(a.z), fast(a.w));
        return make_float4(__fdiv_rn(a.x, b), __fdiv_rn(a.y, b), __fdiv_rn(a.z, b), __fdiv_rn(a.w, b));
    }
};

__device__ __forceinline__ Divisor divisor(float d) { return Divisor{d, __frcp_rn(d), !(fabsf(d) > 9.3132257e-10f && fabsf(d) < 1.0737418e9f)}; }

// A thread's pieces of a channel, `step` elements apart: offsets advance by additions, not by a division per piece.
struct Stride { unsigned rc, z, step, q, r; };              // step = q * rc + r
struct Walk {
    size_t off, gap, hop; unsigned l;
    __device__ __forceinline__ Walk(const Stride &s, unsigned t, unsigned j) {
        const unsigned i = t / s.rc;
        l = t - i * s.rc;
        off = ((size_t)i * s.z + j) * s.rc + l;
        gap = (size_t)(s.z - 1) * s.rc;
        hop = s.step + (size_t)s.q * gap;
    }
    __device__ __forceinline__ void next(const Stride &s) {
        l += s.r; off += hop;
        if (l >= s.rc) { l -= s.rc; off += gap; }
    }
    __device__ __forceinline__ void prev(const Stride &s) {
        off -= hop;
        if (l < s.r) { l += s.rc; off -= gap; }
        l -= s.r;
    }
};
inline Stride stride_of(unsigned z, unsigned rc, unsigned step) { return Stride{rc, z, step, step / rc, step % rc}; }

// The ReLU backward pass folded into the BatchNorm backward pass: delta is src where the layer's output is positive, else 0 (0 + src
// keeps the bits of the separate pass).  MASK 0: no ReLU (src is delta itself); 1: the output is read; 2: it is the
// BatchNorm's own, y = opa * g + b, and is computed again with the roundings of the forward pass instead of being read.
template <int MASK> __device__ __forceinline__ float masked(float d, float o, float i, float g, float b) {
    if (MASK == 0) return d;
    const float y = MASK == 1 ? i : __fadd_rn(__fmul_rn(o, g), b);
    return y > 0.f ? __fadd_rn(0.f, d) : 0.f;
}
template <int MASK> __device__ __forceinline__ float4 masked4(float4 d, float4 o, float4 i, float g, float b) {
    return make_float4(masked<MASK>(d.x, o.x, i.x, g, b), masked<MASK>(d.y, o.y, i.y, g, b), masked<MASK>(d.z, o.z, i.z, g, b), masked<MASK>(d.w, o.w, i.w, g, b));
}

// Terms of sum(d * o), with the roundings spelled out: the compiler's own choice of fused multiply-adds differs between the variants
// with and without a mask, and the folded backward pass has to give the bits of the separate calls.
__device__ __forceinline__ float dot4(float4 d, float4 o) {
    return __fadd_rn(__fmaf_rn(d.x, o.x, __fmul_rn(d.y, o.y)), __fmaf_rn(d.z, o.z, __fmul_rn(d.w, o.w)));
}

// ---- reductions -----------------------------------------------------------------
// MODE 0: (sum x, sum x*x)      MODE 1: (sum d*o, sum d)
template <int MODE, bool VEC, int MASK = 0>
__global__ void __launch_bounds__(kBlock) bn_stats_kernel(const float *__restrict__ x, const float *__restrict__ o,
                                                          float2 *__restrict__ partial, unsigned per, Stride w_,
                                                          const float *__restrict__ act, const float *__restrict__ g, const float *__restrict__ beta) {
    EB_GRID_WAIT();
    __shared__ float sm[32];
    const unsigned j = blockIdx.x, s = blockIdx.y, nsplit = gridDim.y;
    const Slice sl = slice_of(per, nsplit, s);
    float a0 = 0.f, a1 = 0.f;
    const float gj = MASK == 2 ? g[j] : 1.f, bj = MASK == 2 ? beta[j] : 0.f;
    if (VEC) {
        Walk w_at(w_, sl.begin + threadIdx.x * 4, j);
#pragma unroll 4
        for (unsigned t = sl.begin + threadIdx.x * 4; t < sl.end; t += kBlock * 4, w_at.next(w_)) {
            const size_t off = w_at.off;
            float4 v = ldg4(x + off);           // left in L2 on purpose: the apply pass walks its slice backwards
            if (MODE == 0) {
                a0 += (v.x + v.y) + (v.z + v.w);
                a1 += (v.x * v.x + v.y * v.y) + (v.z * v.z + v.w * v.w);
            } else {
                const float4 w = ldg4(o + off);
                if (MASK) v = masked4<MASK>(v, w, MASK == 1 ? ldg4(act + off) : w, gj, bj);
                a0 = __fadd_rn(a0, dot4(v, w));
                a1 += (v.x + v.y) + (v.z + v.w);
            }
        }
    } else {
        Walk w_at(w_, sl.begin + threadIdx.x, j);
        for (unsigned t = sl.begin + threadIdx.x; t < sl.end; t += kBlock, w_at.next(w_)) {
            const size_t off = w_at.off;
            float v = x[off];
            if (MODE == 0) { a0 += v; a1 += v * v; }
            else {
                const float w = o[off];
                if (MASK) v = masked<MASK>(v, w, MASK == 1 ? act[off] : w, gj, bj);
                a0 = __fmaf_rn(v, w, a0); a1 += v;
            }
        }
    }
    a0 = block_sum(a0, sm);
    a1 = block_sum(a1, sm);
    if (threadIdx.x == 0) partial[(size_t)j * nsplit + s] = make_float2(a0, a1);
}

__device__ __forceinline__ void reduce_partials(const float2 *partial, unsigned j, unsigned nsplit, float *sh, float &s0, float &s1) {
    // nsplit <= kMaxSplit <= blockDim.x ; combine in double, round once
    double d0 = 0.0, d1 = 0.0;
    if (threadIdx.x < 32) {
        for (unsigned s = threadIdx.x; s < nsplit; s += 32) {
            const float2 p = partial[(size_t)j * nsplit + s];
            d0 += (double)p.x; d1 += (double)p.y;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            d0 += __shfl_xor_sync(0xffffffffu, d0, o);
            d1 += __shfl_xor_sync(0xffffffffu, d1, o);
        }
        if (threadIdx.x == 0) { sh[0] = (float)d0; sh[1] = (float)d1; }
    }
    __syncthreads();
    s0 = sh[0]; s1 = sh[1];
}

// ---- forward apply ----------------------------------------------------------------
template <bool TRAIN, bool VEC>
__global__ void __launch_bounds__(kBlock) bn_fwd_apply_kernel(const float *__restrict__ x, float *__restrict__ y, float *__restrict__ opa,
                                                              float *__restrict__ relu_out,
                                                              const float2 *__restrict__ partial,
                                                              float *global_mean, float *global_var,
                                                              const float *__restrict__ g, const float *__restrict__ beta,
                                                              float *mean_out, float *var_out,
                                                              unsigned per, Stride w_, float eps, float momentum) {
    EB_GRID_WAIT();
    __shared__ float sh[2];
    // slices in reverse launch order: the statistics pass finished with the highest slices, so those are what the L2 holds
    const unsigned j = blockIdx.x, nsplit = gridDim.y, s = nsplit - 1 - blockIdx.y;
    float mean, sigma;
    if (TRAIN) {
        float sum, sumsq;
        reduce_partials(partial, j, nsplit, sh, sum, sumsq);
        const float N = (float)per;                                    // float N = b * rc;
        mean = __fdiv_rn(sum, N);                                      // mean[j] / N
        const float var = __fsub_rn(__fdiv_rn(sumsq, N), __fmul_rn(mean, mean));
        sigma = __fsqrt_rn(__fadd_rn(var, eps));                       // sqrt(variance[j] + epsilon)
        if (s == 0 && threadIdx.x == 0) {
            if (momentum != 0.0f) {
                // momentum * global[j] is a float product; (1.0 - momentum) * stat is double
                const double keep = 1.0 - (double)momentum;
                global_mean[j] = (float)((double)__fmul_rn(momentum, global_mean[j]) + keep * (double)mean);
                global_var[j] = (float)((double)__fmul_rn(momentum, global_var[j]) + keep * (double)var);
            }
            mean_out[j] = mean;
            var_out[j] = sigma;
        }
    } else {
        mean = global_mean[j];
        sigma = __fsqrt_rn(__fadd_rn(global_var[j], eps));
        if (s == 0 && threadIdx.x == 0) var_out[j] = sigma;
    }
    const bool affine = (g != nullptr);
    const float gj = affine ? g[j] : 1.f, bj = affine ? beta[j] : 0.f;
    const Slice sl = slice_of(per, nsplit, s);
    const Divisor div = divisor(sigma);
    if (VEC) {
        const unsigned first = sl.begin + threadIdx.x * 4, pieces = first < sl.end ? (sl.end - first + kBlock * 4 - 1) / (kBlock * 4) : 0;
        if (!pieces) return;
        Walk at(w_, first + (pieces - 1) * (kBlock * 4), j);
#pragma unroll 4
        // Backwards through the slice: the statistics pass read it forwards just before, so its tail is what the L2 still
        // holds; the second read of tensors up to about the L2 size then costs no HBM traffic.
        for (unsigned it = pieces; it-- > 0; at.prev(w_)) {
            const size_t off = at.off;
            const float4 v = ld_stream4(x + off);
            float4 o, r;
            o = div(make_float4(__fsub_rn(v.x, mean), __fsub_rn(v.y, mean), __fsub_rn(v.z, mean), __fsub_rn(v.w, mean)));
            if (affine) {
                *reinterpret_cast<float4 *>(opa + off) = o;
                r.x = __fadd_rn(__fmul_rn(o.x, gj), bj); r.y = __fadd_rn(__fmul_rn(o.y, gj), bj);
                r.z = __fadd_rn(__fmul_rn(o.z, gj), bj); r.w = __fadd_rn(__fmul_rn(o.w, gj), bj);
            } else {
                r = o;
            }
            *reinterpret_cast<float4 *>(y + off) = r;
            if (relu_out) {
                r.x = r.x > 0.f ? r.x : 0.f; r.y = r.y > 0.f ? r.y : 0.f; r.z = r.z > 0.f ? r.z : 0.f; r.w = r.w > 0.f ? r.w : 0.f;
                *reinterpret_cast<float4 *>(relu_out + off) = r;
            }
        }
    } else {
        const unsigned first = sl.begin + threadIdx.x, pieces = first < sl.end ? (sl.end - first + kBlock - 1) / kBlock : 0;
        if (!pieces) return;
        Walk at(w_, first + (pieces - 1) * kBlock, j);
        for (unsigned it = pieces; it-- > 0; at.prev(w_)) {
            const size_t off = at.off;
            const float o = div(__fsub_rn(x[off], mean));
            float r = o;
            if (affine) { opa[off] = o; r = __fadd_rn(__fmul_rn(o, gj), bj); }
            y[off] = r;
            if (relu_out) relu_out[off] = r > 0.f ? r : 0.f;
        }
    }
}

// ---- backward apply ---------------------------------------------------------------
// PD_ZERO: the parent delta is known to hold zeros, so it is written without being read (0 + x keeps the bits of the
// read-modify-write form).
template <bool VEC, bool PD_ZERO, int MASK = 0>
__global__ void __launch_bounds__(kBlock) bn_bwd_apply_kernel(float *__restrict__ delta, const float *__restrict__ opa, float *__restrict__ pdelta,
                                                              const float *__restrict__ src, const float *__restrict__ act, const float *__restrict__ beta,
                                                              const float2 *__restrict__ partial,
                                                              float *gbn_g, float *gbn_b, const float *__restrict__ bn_g,
                                                              const float *__restrict__ variance, float *mean1, float *mean2,
                                                              unsigned per, Stride w_) {
    EB_GRID_WAIT();
    __shared__ float sh[2];
    const unsigned j = blockIdx.x, nsplit = gridDim.y, s = nsplit - 1 - blockIdx.y;     // reverse launch order, see forward
    float s1, s2;
    reduce_partials(partial, j, nsplit, sh, s1, s2);
    const float N = (float)per;
    float m1 = __fdiv_rn(s1, N), m2 = __fdiv_rn(s2, N);
    const bool affine = (bn_g != nullptr);
    const float gj = affine ? bn_g[j] : 1.f, bj = MASK == 2 ? beta[j] : 0.f;
    if (s == 0 && threadIdx.x == 0 && affine) {
        gbn_g[j] = __fadd_rn(gbn_g[j], m1);      // gradients of gamma/beta are MEANS in the reference
        gbn_b[j] = __fadd_rn(gbn_b[j], m2);
    }
    if (affine) { m1 = __fmul_rn(m1, gj); m2 = __fmul_rn(m2, gj); }
    if (s == 0 && threadIdx.x == 0) { mean1[j] = m1; mean2[j] = m2; }
    const float sigma = variance[j];
    const Slice sl = slice_of(per, nsplit, s);
    const Divisor div = divisor(sigma);
    if (VEC) {
        const unsigned first = sl.begin + threadIdx.x * 4, pieces = first < sl.end ? (sl.end - first + kBlock * 4 - 1) / (kBlock * 4) : 0;
        if (!pieces) return;
        Walk at(w_, first + (pieces - 1) * (kBlock * 4), j);
#pragma unroll 4
        // Backwards through the slice: the statistics pass read it forwards just before, so its tail is what the L2 still
        // holds; the second read of tensors up to about the L2 size then costs no HBM traffic.
        for (unsigned it = pieces; it-- > 0; at.prev(w_)) {
            const size_t off = at.off;
            float4 d = MASK ? ld_stream4(src + off) : *reinterpret_cast<const float4 *>(delta + off);
            const float4 o = ld_stream4(opa + off);
            if (MASK) d = masked4<MASK>(d, o, MASK == 1 ? ld_stream4(act + off) : o, gj, bj);
            float4 p = PD_ZERO ? make_float4(0.f, 0.f, 0.f, 0.f) : *reinterpret_cast<const float4 *>(pdelta + off);
            if (affine) {
                d.x = __fmul_rn(d.x, gj); d.y = __fmul_rn(d.y, gj); d.z = __fmul_rn(d.z, gj); d.w = __fmul_rn(d.w, gj);
                *reinterpret_cast<float4 *>(delta + off) = d;            // delta[p] *= bn_g[j]
            } else if (MASK) *reinterpret_cast<float4 *>(delta + off) = d;
            const float4 q = div(make_float4(__fsub_rn(d.x, __fadd_rn(__fmul_rn(o.x, m1), m2)), __fsub_rn(d.y, __fadd_rn(__fmul_rn(o.y, m1), m2)),
                                             __fsub_rn(d.z, __fadd_rn(__fmul_rn(o.z, m1), m2)), __fsub_rn(d.w, __fadd_rn(__fmul_rn(o.w, m1), m2))));
            p.x = __fadd_rn(p.x, q.x); p.y = __fadd_rn(p.y, q.y); p.z = __fadd_rn(p.z, q.z); p.w = __fadd_rn(p.w, q.w);
            *reinterpret_cast<float4 *>(pdelta + off) = p;
        }
    } else {
        const unsigned first = sl.begin + threadIdx.x, pieces = first < sl.end ? (sl.end - first + kBlock - 1) / kBlock : 0;
        if (!pieces) return;
        Walk at(w_, first + (pieces - 1) * kBlock, j);
        for (unsigned it = pieces; it-- > 0; at.prev(w_)) {
            const size_t off = at.off;
            const float o = opa[off];
            float d = MASK ? masked<MASK>(src[off], o, MASK == 1 ? act[off] : o, gj, bj) : delta[off];
            if (affine) d = __fmul_rn(d, gj);
            if (affine || MASK) delta[off] = d;
            pdelta[off] = __fadd_rn(PD_ZERO ? 0.f : pdelta[off], div(__fsub_rn(d, __fadd_rn(__fmul_rn(o, m1), m2))));
        }
    }
}

// ---- one launch: channels in the shared memory of clusters ---------------------------------------------
// Small and middle-sized tensors: a channel is spread over the blocks of a cluster (one block for small planes), which keep their
// shares in shared memory; each adds up its part of the sums, the blocks exchange them through distributed shared memory (added
// in rank order, in double) and write their outputs -- one launch instead of two, every element read once.  A cluster walks over
// channels (persistent grid): the copies of the next channel into a second buffer (cp.async) run while this one is reduced
// and written, and a thread only reads pieces that it has copied itself, so there is no barrier between copy and use.
// 128 x 512 x 4 x 4: forward 7.4 -> 4.5 us; 64 x 256 x 14 x 14: 14.4 -> 9.9.  Large tensors stay with two passes (see one_plan):
// those run at what HBM gives for their traffic (64 x 256 x 56 x 56 backward: 1.23 GB in 203 us), while here a block stalls in
// every channel until the slowest block of its cluster has its data (332 us although a third less is moved).
constexpr int kOneBlock = 1024;

__device__ __forceinline__ void copy_async(float *dst, const float *src, bool wide) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if (wide) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

struct OneCut { unsigned per, chunk, csize, clusters; Stride w; };             // how a channel is cut

// Sums over the cluster (the block alone when csize is 1).
__device__ __forceinline__ float2 cluster_totals(float a0, float a1, unsigned csize, float *sm, float2 *slot, float2 *total) {
    a0 = block_sum(a0, sm);
    a1 = block_sum(a1, sm);
    if (csize == 1) return make_float2(a0, a1);
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    if (threadIdx.x == 0) *slot = make_float2(a0, a1);
    cluster.sync();
    if (threadIdx.x < 32) {
        double d0 = 0.0, d1 = 0.0;
        if (threadIdx.x < csize) { const float2 p = *cluster.map_shared_rank(slot, threadIdx.x); d0 = p.x; d1 = p.y; }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) { d0 += __shfl_xor_sync(0xffffffffu, d0, o); d1 += __shfl_xor_sync(0xffffffffu, d1, o); }
        if (threadIdx.x == 0) *total = make_float2((float)d0, (float)d1);
    }
    __syncthreads();
    return *total;
}

template <bool VEC>
__global__ void __launch_bounds__(kOneBlock) bn_fwd_one_kernel(const float *__restrict__ x, float *__restrict__ y, float *__restrict__ opa, float *__restrict__ relu_out,
                                                               float *global_mean, float *global_var, const float *__restrict__ g, const float *__restrict__ beta,
                                                               float *mean_out, float *var_out, OneCut c, float eps, float momentum) {
    extern __shared__ __align__(16) float buf[];
    __shared__ float sm[32];
    __shared__ float2 slot[2], total[2];
    EB_GRID_WAIT();
    constexpr unsigned V = VEC ? 4 : 1;
    const unsigned cluster = blockIdx.x / c.csize, rank = blockIdx.x - cluster * c.csize;
    const unsigned begin = min(rank * c.chunk, c.per), n = min(c.chunk, c.per - begin);
    auto fetch = [&](unsigned j, float *dst) {
        Walk w(c.w, begin + threadIdx.x * V, j);
        for (unsigned t = threadIdx.x * V; t < n; t += c.w.step, w.next(c.w)) copy_async(dst + t, x + w.off, VEC);
        copy_commit();
    };
    if (cluster < c.w.z) fetch(cluster, buf);
    unsigned k = 0;
    for (unsigned j = cluster; j < c.w.z; j += c.clusters, k++) {
        float *cur = buf + (k & 1) * c.chunk;
        if (j + c.clusters < c.w.z) fetch(j + c.clusters, buf + ((k + 1) & 1) * c.chunk); else copy_commit();
        copy_wait<1>();
        float a0 = 0.f, a1 = 0.f;
#pragma unroll 4
        for (unsigned t = threadIdx.x * V; t < n; t += c.w.step) {
            if (VEC) {
                const float4 v = *reinterpret_cast<const float4 *>(cur + t);
                a0 += (v.x + v.y) + (v.z + v.w);
                a1 += (v.x * v.x + v.y * v.y) + (v.z * v.z + v.w * v.w);
            } else { const float v = cur[t]; a0 += v; a1 += v * v; }
        }
        const float2 sum = cluster_totals(a0, a1, c.csize, sm, slot + (k & 1), total + (k & 1));
        const float N = (float)c.per;                                          // float N = b * rc;
        const float mean = __fdiv_rn(sum.x, N);                                // mean[j] / N
        const float var = __fsub_rn(__fdiv_rn(sum.y, N), __fmul_rn(mean, mean));
        const float sigma = __fsqrt_rn(__fadd_rn(var, eps));                   // sqrt(variance[j] + epsilon)
        if (rank == 0 && threadIdx.x == 0) {
            if (momentum != 0.0f) {
                // momentum * global[j] is a float product; (1.0 - momentum) * stat is double
                const double keep = 1.0 - (double)momentum;
                global_mean[j] = (float)((double)__fmul_rn(momentum, global_mean[j]) + keep * (double)mean);
                global_var[j] = (float)((double)__fmul_rn(momentum, global_var[j]) + keep * (double)var);
            }
            mean_out[j] = mean;
            var_out[j] = sigma;
        }
        const bool affine = (g != nullptr);
        const float gj = affine ? g[j] : 1.f, bj = affine ? beta[j] : 0.f;
        const Divisor div = divisor(sigma);
        Walk w(c.w, begin + threadIdx.x * V, j);
#pragma unroll 2
        for (unsigned t = threadIdx.x * V; t < n; t += c.w.step, w.next(c.w)) {
            const size_t off = w.off;
            if (VEC) {
                const float4 v = *reinterpret_cast<const float4 *>(cur + t);
                float4 o, r;
                o = div(make_float4(__fsub_rn(v.x, mean), __fsub_rn(v.y, mean), __fsub_rn(v.z, mean), __fsub_rn(v.w, mean)));
                r = o;
                if (affine) {
                    *reinterpret_cast<float4 *>(opa + off) = o;
                    r.x = __fadd_rn(__fmul_rn(o.x, gj), bj); r.y = __fadd_rn(__fmul_rn(o.y, gj), bj);
                    r.z = __fadd_rn(__fmul_rn(o.z, gj), bj); r.w = __fadd_rn(__fmul_rn(o.w, gj), bj);
                }
                *reinterpret_cast<float4 *>(y + off) = r;
                if (relu_out) {
                    r.x = r.x > 0.f ? r.x : 0.f; r.y = r.y > 0.f ? r.y : 0.f; r.z = r.z > 0.f ? r.z : 0.f; r.w = r.w > 0.f ? r.w : 0.f;
                    *reinterpret_cast<float4 *>(relu_out + off) = r;
                }
            } else {
                const float o = div(__fsub_rn(cur[t], mean));
                float r = o;
                if (affine) { opa[off] = o; r = __fadd_rn(__fmul_rn(o, gj), bj); }
                y[off] = r;
                if (relu_out) relu_out[off] = r > 0.f ? r : 0.f;
            }
        }
    }
    if (c.csize > 1) cooperative_groups::this_cluster().sync();        // the others may still read this block's slot
}

template <bool VEC, bool PD_ZERO, int MASK>
__global__ void __launch_bounds__(kOneBlock) bn_bwd_one_kernel(float *delta, const float *__restrict__ opa, float *__restrict__ pdelta,
                                                               const float *src, const float *__restrict__ act, const float *__restrict__ beta,
                                                               float *gbn_g, float *gbn_b, const float *__restrict__ bn_g, const float *__restrict__ variance,
                                                               float *mean1, float *mean2, OneCut c) {
    extern __shared__ __align__(16) float buf[];
    __shared__ float sm[32];
    __shared__ float2 slot[2], total[2];
    EB_GRID_WAIT();
    constexpr unsigned V = VEC ? 4 : 1;
    constexpr unsigned TENSORS = MASK == 1 ? 3 : 2;
    const unsigned cluster = blockIdx.x / c.csize, rank = blockIdx.x - cluster * c.csize;
    const unsigned begin = min(rank * c.chunk, c.per), n = min(c.chunk, c.per - begin);
    const bool affine = (bn_g != nullptr);
    auto fetch = [&](unsigned j, float *dst) {
        Walk w(c.w, begin + threadIdx.x * V, j);
        for (unsigned t = threadIdx.x * V; t < n; t += c.w.step, w.next(c.w)) {
            copy_async(dst + t, src + w.off, VEC);
            copy_async(dst + c.chunk + t, opa + w.off, VEC);
            if (MASK == 1) copy_async(dst + 2 * c.chunk + t, act + w.off, VEC);
        }
        copy_commit();
    };
    if (cluster < c.w.z) fetch(cluster, buf);
    unsigned k = 0;
    for (unsigned j = cluster; j < c.w.z; j += c.clusters, k++) {
        float *bd = buf + (k & 1) * (TENSORS * c.chunk), *bo = bd + c.chunk, *ba = bo + c.chunk;
        if (j + c.clusters < c.w.z) fetch(j + c.clusters, buf + ((k + 1) & 1) * (TENSORS * c.chunk)); else copy_commit();
        const float gj = affine ? bn_g[j] : 1.f, bj = MASK == 2 ? beta[j] : 0.f;
        copy_wait<1>();
        float a0 = 0.f, a1 = 0.f;
#pragma unroll 4
        for (unsigned t = threadIdx.x * V; t < n; t += c.w.step) {
            if (VEC) {
                float4 v = *reinterpret_cast<const float4 *>(bd + t);
                const float4 w = *reinterpret_cast<const float4 *>(bo + t);
                if (MASK) { v = masked4<MASK>(v, w, MASK == 1 ? *reinterpret_cast<const float4 *>(ba + t) : w, gj, bj); *reinterpret_cast<float4 *>(bd + t) = v; }
                a0 = __fadd_rn(a0, dot4(v, w));
                a1 += (v.x + v.y) + (v.z + v.w);
            } else {
                float v = bd[t];
                const float w = bo[t];
                if (MASK) { v = masked<MASK>(v, w, MASK == 1 ? ba[t] : w, gj, bj); bd[t] = v; }
                a0 = __fmaf_rn(v, w, a0); a1 += v;
            }
        }
        const float2 sum = cluster_totals(a0, a1, c.csize, sm, slot + (k & 1), total + (k & 1));
        const float N = (float)c.per;
        float m1 = __fdiv_rn(sum.x, N), m2 = __fdiv_rn(sum.y, N);
        if (rank == 0 && threadIdx.x == 0 && affine) {
            gbn_g[j] = __fadd_rn(gbn_g[j], m1);      // gradients of gamma/beta are MEANS in the reference
            gbn_b[j] = __fadd_rn(gbn_b[j], m2);
        }
        if (affine) { m1 = __fmul_rn(m1, gj); m2 = __fmul_rn(m2, gj); }
        if (rank == 0 && threadIdx.x == 0) { mean1[j] = m1; mean2[j] = m2; }
        const float sigma = variance[j];
        const Divisor div = divisor(sigma);
        auto rest = [&](float d, float o) { return __fsub_rn(d, __fadd_rn(__fmul_rn(o, m1), m2)); };
        Walk w(c.w, begin + threadIdx.x * V, j);
#pragma unroll 2
        for (unsigned t = threadIdx.x * V; t < n; t += c.w.step, w.next(c.w)) {
            const size_t off = w.off;
            if (VEC) {
                float4 d = *reinterpret_cast<const float4 *>(bd + t);
                const float4 o = *reinterpret_cast<const float4 *>(bo + t);
                float4 p = PD_ZERO ? make_float4(0.f, 0.f, 0.f, 0.f) : *reinterpret_cast<const float4 *>(pdelta + off);
                if (affine) { d.x = __fmul_rn(d.x, gj); d.y = __fmul_rn(d.y, gj); d.z = __fmul_rn(d.z, gj); d.w = __fmul_rn(d.w, gj); }
                if (affine || MASK) *reinterpret_cast<float4 *>(delta + off) = d;            // delta[p] *= bn_g[j]
                const float4 q = div(make_float4(rest(d.x, o.x), rest(d.y, o.y), rest(d.z, o.z), rest(d.w, o.w)));
                p.x = __fadd_rn(p.x, q.x); p.y = __fadd_rn(p.y, q.y); p.z = __fadd_rn(p.z, q.z); p.w = __fadd_rn(p.w, q.w);
                *reinterpret_cast<float4 *>(pdelta + off) = p;
            } else {
                float d = bd[t];
                if (affine) d = __fmul_rn(d, gj);
                if (affine || MASK) delta[off] = d;
                pdelta[off] = __fadd_rn(PD_ZERO ? 0.f : pdelta[off], div(rest(d, bo[t])));
            }
        }
    }
    if (c.csize > 1) cooperative_groups::this_cluster().sync();        // the others may still read this block's slot
}

// Cluster size, block size and grid for channels of `per` elements with `tensors` of them in shared memory, twice (this channel and
// the next).  Small channels: one block each, as many blocks as fit an SM.  Larger ones are spread over up to 16 blocks, two of
// them per SM where that is enough (one block's copies and stores run while the other exchanges sums), else one.
// false = the two-pass kernels: the channel does not fit, or it needs a cluster and the tensor is larger than 8 MB (the backward
// pass, with twice the shared memory per element, from there on in any case): measured at 0.2 to 200 MB.
struct OnePlan { OneCut c; unsigned threads, smem, blocks; };
bool one_plan(unsigned z, unsigned per, unsigned rc, int tensors, bool vec, OnePlan &p) {
    const size_t bytes = (size_t)per * 4 * tensors * 2, two = 112 * 1024, one = 224 * 1024;
    unsigned cs = 1;
    while (cs < 16 && bytes > two * cs) cs *= 2;
    // few channels: cut finer until every SM has work (shares of at least 1024 elements)
    while (cs < 16 && (size_t)z * cs < EDDLB200_NUM_SMS && per >= 2 * cs * 1024) cs *= 2;
    OneCut &c = p.c;
    c.per = per; c.csize = cs;
    c.chunk = ((per + cs - 1) / cs + 3u) & ~3u;
    p.smem = c.chunk * 4 * tensors * 2;
    if (p.smem > one) return false;
    // about four pieces per thread; 32 warps per SM for the large shares
    const unsigned want = c.chunk / (vec ? 16 : 4);
    p.threads = p.smem > two ? 1024 : want >= 512 ? 512 : want >= 256 ? 256 : want >= 128 ? 128 : 64;
    unsigned per_sm = (unsigned)(one / (p.smem + 1024));
    if (per_sm > 1536 / p.threads) per_sm = 1536 / p.threads;
    if (per_sm > 16) per_sm = 16;
    if (per_sm < 1) per_sm = 1;
    c.clusters = EDDLB200_NUM_SMS * per_sm / cs;
    if (c.clusters > z) c.clusters = z;
    p.blocks = c.clusters * cs;
    c.w = stride_of(z, rc, p.threads * (vec ? 4 : 1));
    if ((size_t)z * per * 4 > (size_t)8 << 20 && (cs > 1 || tensors > 1)) return false;
    return true;
}
// What a kernel has been set up for on one device.
struct OneSetup { std::atomic<bool> attributes{false}; std::atomic<unsigned> wide_smem{0}; };        // wide_smem: shared memory known to fit clusters of 16
// kNotTaken where the device cannot hold a cluster of this size (more than eight blocks are not guaranteed: a 16-block cluster needs
// that many SMs of one cluster group free of other limits); a launch that fails for any other reason is an error.
template <typename... P, typename... A>
int launch_one(void (*kernel)(P...), OneSetup &setup, const OnePlan &p, cudaStream_t st, A &&...args) {
    if (!setup.attributes) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return cuda_status(e, "gpu_batchnorm(attributes)");
        setup.attributes = true;
    }
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension; at[0].val.clusterDim.x = p.c.csize; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.blocks); cfg.blockDim = dim3(p.threads); cfg.dynamicSmemBytes = p.smem; cfg.stream = st; cfg.attrs = at; cfg.numAttrs = 2;
    if (p.c.csize > 8 && p.smem > setup.wide_smem) {
        cudaLaunchConfig_t query = cfg;
        query.blockDim = dim3(kOneBlock); query.numAttrs = 1;              // the largest block: what fits it fits the smaller ones
        int clusters = 0;
        cudaError_t e = cudaOccupancyMaxActiveClusters(&clusters, kernel, &query);
        if (e != cudaSuccess || clusters < 1) { cudaGetLastError(); return kNotTaken; }
        setup.wide_smem = p.smem;
    }
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
    return cuda_status(cudaGetLastError(), "gpu_batchnorm(one launch)");
}

// Training-mode forward in one launch; kNotTaken = the caller takes the two-pass kernels.
int fwd_one_launch(int dev, cudaStream_t st, unsigned b, unsigned z, unsigned rc, bool vec, const float *input, float *output, float *opa, float *global_mean, float *global_variance,
                   const float *affine_g, const float *affine_b, float *mean, float *variance, float epsilon, float momentum, float *relu_out) {
    OnePlan p;
    if (!one_plan(z, b * rc, rc, 1, vec, p)) return kNotTaken;
    static OneSetup setup[EDDLB200_MAX_DEVICES][2];
    return launch_one(vec ? bn_fwd_one_kernel<true> : bn_fwd_one_kernel<false>, setup[dev][vec], p, st, input, output, opa, relu_out, global_mean, global_variance,
                      affine_g, affine_b, mean, variance, p.c, epsilon, momentum);
}

template <bool PD_ZERO, int MASK>
int bwd_one_launch(int dev, cudaStream_t st, unsigned b, unsigned z, unsigned rc, bool vec, float *delta, const float *opa, float *pdelta, const float *src, const float *act,
                   const float *beta, float *gbn_g, float *gbn_b, const float *bn_g, const float *variance, float *mean1, float *mean2) {
    OnePlan p;
    if (!one_plan(z, b * rc, rc, MASK == 1 ? 3 : 2, vec, p)) return kNotTaken;
    static OneSetup setup[EDDLB200_MAX_DEVICES][2];
    return launch_one(vec ? bn_bwd_one_kernel<true, PD_ZERO, MASK> : bn_bwd_one_kernel<false, PD_ZERO, MASK>, setup[dev][vec], p, st, delta, opa, pdelta, src, act,
                      beta, gbn_g, gbn_b, bn_g, variance, mean1, mean2, p.c);
}

void fwd_two_pass(cudaStream_t st, unsigned S, bool vec, const float *input, float *output, float *opa, float *relu_out, float2 *partial, float *global_mean, float *global_variance,
                  const float *affine_g, const float *affine_b, float *mean, float *variance, unsigned z, unsigned rc, unsigned per, float epsilon, float momentum) {
    const Stride w = stride_of(z, rc, vec ? kBlock * 4 : kBlock);
    const dim3 grid(z, S);
    eb::launch(vec ? bn_stats_kernel<0, true> : bn_stats_kernel<0, false>, grid, kBlock, 0, st, input, nullptr, partial, per, w, nullptr, nullptr, nullptr);
    eb::launch(vec ? bn_fwd_apply_kernel<true, true> : bn_fwd_apply_kernel<true, false>, grid, kBlock, 0, st, input, output, opa, relu_out, partial, global_mean, global_variance,
               affine_g, affine_b, mean, variance, per, w, epsilon, momentum);
}

template <bool PD_ZERO, int MASK>
void bwd_two_pass(cudaStream_t st, unsigned S, bool vec, float *delta, const float *opa, float *pdelta, const float *src, const float *act, const float *beta, float2 *partial,
                  float *gbn_g, float *gbn_b, const float *bn_g, const float *variance, float *mean1, float *mean2, unsigned b, unsigned z, unsigned rc) {
    const Stride w = stride_of(z, rc, vec ? kBlock * 4 : kBlock);
    const dim3 grid(z, S);
    eb::launch(vec ? bn_stats_kernel<1, true, MASK> : bn_stats_kernel<1, false, MASK>, grid, kBlock, 0, st, src, opa, partial, b * rc, w, act, bn_g, beta);
    eb::launch(vec ? bn_bwd_apply_kernel<true, PD_ZERO, MASK> : bn_bwd_apply_kernel<false, PD_ZERO, MASK>, grid, kBlock, 0, st, delta, opa, pdelta, src, act, beta, partial,
               gbn_g, gbn_b, bn_g, variance, mean1, mean2, b * rc, w);
}

// Slices per channel.  A launch is cut into several waves of short-lived blocks (g_bn_waves times the 8 blocks of 256 threads
// an SM holds): with barely more blocks than the GPU holds at once, the few left over for a second wave run almost alone
// at a fraction of the bandwidth while the rest of the GPU idles.
int g_bn_waves = 16, g_bn_min_items = 8192;
inline unsigned pick_split(unsigned z, unsigned per_channel) {
    unsigned want = (EDDLB200_NUM_SMS * 8 * (unsigned)g_bn_waves + z - 1) / z;
    unsigned cap = (per_channel + (unsigned)g_bn_min_items - 1) / (unsigned)g_bn_min_items;
    unsigned s = want < cap ? want : cap;
    if (s < 1) s = 1;
    if (s > kMaxSplit) s = kMaxSplit;
    return s;
}

// Whether a ReLU backward pass is folded in: not where the two-pass kernels go element by element (planes that are no multiple of
// four long, unaligned tensors).  Every element then costs three or four 4-byte loads in each pass, and the separate ReLU pass,
// which does not care about planes, is the cheaper one: 64 x 64 x 27 x 27 48 us folded, 36 separate.  Short planes in many
// channels of one slice are the exception (64 x 1024 x 7 x 7 28 and 32).  With 16-byte loads 64 x 512 x 28 x 28 takes 111 to 140 us
// folded, 155 separate.
bool fold_pays(unsigned z, unsigned per, unsigned rc, int tensors, bool vec) {
    OnePlan p;
    return vec || one_plan(z, per, rc, tensors, vec, p) || (rc < 64 && z >= 512 && pick_split(z, per) == 1);
}

}  // namespace

namespace eb {
// tuning knobs behind eddlb200_set_option("bn_waves" / "bn_min_items")
int bn_set_tuning(int waves, int min_items) {
    if (waves > 0) g_bn_waves = waves > 64 ? 64 : waves;
    if (min_items > 0) g_bn_min_items = min_items < 1024 ? 1024 : min_items;
    return 0;
}
}  // namespace eb

using namespace eb;

extern "C" {

int eddlb200_bn_fwd(int dev, int b, int z, int rc, const float *input, float *output, float *opa,
                    float *global_mean, float *global_variance, const float *affine_g, const float *affine_b,
                    float *mean, float *variance, int trmode, float epsilon, float momentum, float *relu_out) {
    EB_CTX(dev);
    EB_REQUIRE(b > 0 && z > 0 && rc > 0 && input && output && global_mean && global_variance && variance, "gpu_batchnorm_forward");
    EB_REQUIRE((size_t)b * rc < 0xfffffff0u, "gpu_batchnorm_forward");
    EB_REQUIRE(!affine_g || (affine_b && opa), "gpu_batchnorm_forward");
    EB_REQUIRE(!trmode || mean, "gpu_batchnorm_forward");
    {
        const size_t tb = (size_t)b * z * rc * sizeof(float), zb = (size_t)z * sizeof(float);
        EB_READS(input, tb); EB_WRITES(output, tb); EB_WRITES(opa, tb); EB_WRITES(relu_out, tb);
        EB_MODIFIES(global_mean, zb); EB_MODIFIES(global_variance, zb); EB_READS(affine_g, zb); EB_READS(affine_b, zb);
        EB_MODIFIES(mean, zb); EB_MODIFIES(variance, zb);
    }
    // bytes per element: x, y, and the two optional outputs -- opa (the normalised value BN backward needs) and the ReLU of y
    // written for the layer that follows
    ProfScope prof(cx, PROF_BN_FWD, (4.0 + 4.0 + (opa ? 4.0 : 0.0) + (relu_out ? 4.0 : 0.0)) * b * (double)z * rc);
    const unsigned per = (unsigned)b * rc, S = pick_split(z, per);
    const bool vec = (rc % 4 == 0) && aligned16(input) && aligned16(output) && (!opa || aligned16(opa)) && (!relu_out || aligned16(relu_out));
    const Stride w = stride_of(z, rc, vec ? kBlock * 4 : kBlock);
    dim3 grid(z, S);
    float2 *partial = nullptr;
    if (trmode && affine_g && opa && lz_enabled(cx)) bn_source_set(cx, output, opa, affine_g, affine_b, (size_t)b * z * rc, z, rc);
    if (trmode) {
        const int r = fwd_one_launch(dev, st, b, z, rc, vec, input, output, opa, global_mean, global_variance, affine_g, affine_b, mean, variance, epsilon, momentum, relu_out);
        if (r == 0) count_launch(cx);
        if (r != kNotTaken) return r;
        partial = (float2 *)scratch(cx, (size_t)z * S * sizeof(float2));
        if (!partial) return cudaErrorMemoryAllocation;
        fwd_two_pass(st, S, vec, input, output, opa, relu_out, partial, global_mean, global_variance, affine_g, affine_b, mean, variance, z, rc, per, epsilon, momentum);
        count_launch(cx);
    } else {
        if (vec) eb::launch(bn_fwd_apply_kernel<false, true>, grid, kBlock, 0, st, input, output, opa, relu_out, nullptr, global_mean, global_variance, affine_g, affine_b, mean, variance, per, w, epsilon, momentum);
        else eb::launch(bn_fwd_apply_kernel<false, false>, grid, kBlock, 0, st, input, output, opa, relu_out, nullptr, global_mean, global_variance, affine_g, affine_b, mean, variance, per, w, epsilon, momentum);
    }
    EB_LAUNCH_CHECK("gpu_batchnorm_forward(apply)");
    return 0;
}

int eddlb200_bn_bwd(int dev, int b, int z, int rc, float *delta, const float *opa, float *pdelta,
                    float *gbn_g, float *gbn_b, const float *bn_g, const float *variance, float *mean1, float *mean2) {
    EB_CTX_KEEP_PENDING(dev);
    EB_REQUIRE(b > 0 && z > 0 && rc > 0 && delta && opa && pdelta && variance && mean1 && mean2, "gpu_batchnorm_backward");
    EB_REQUIRE((size_t)b * rc < 0xfffffff0u, "gpu_batchnorm_backward");
    EB_REQUIRE(!bn_g || (gbn_g && gbn_b), "gpu_batchnorm_backward");
    const size_t elements = (size_t)b * z * rc;
    const float *src = delta, *act = nullptr, *beta = nullptr;
    int mask = 0;
    if (pend_copy_active(cx)) {
        PendCopy &p = pend_copy(cx);
        // what the fold reads after the call has begun to write: the two inputs of the ReLU backward pass, which a caller may give
        // up (and use again for an output) once that pass has been called
        bool apart = pdelta != delta;
        for (const float *in : {p.src, p.src2}) {
            const size_t tb = elements * sizeof(float), zb = (size_t)z * sizeof(float);
            apart = apart && !overlap(in, tb, pdelta, tb) && !overlap(in, tb, gbn_g, zb) && !overlap(in, tb, gbn_b, zb) && !overlap(in, tb, mean1, zb) && !overlap(in, tb, mean2, zb);
        }
        const float *own = nullptr;                                      // beta, where what ReLU tests can be computed again
        if (p.kind == 4 && p.dst == delta && p.n == elements && apart) own = bn_g ? bn_source_beta(cx, p.src2, opa, bn_g, elements, z, rc) : nullptr;
        if (p.kind == 4 && p.dst == delta && p.n == elements && apart &&
            fold_pays(z, (unsigned)b * rc, rc, own ? 2 : 3, rc % 4 == 0 && aligned16(delta) && aligned16(opa) && aligned16(pdelta) && aligned16(p.src) && (own || aligned16(p.src2)))) {
            // the ReLU backward pass that makes this delta is still on record: it is folded in
            p.active = false;
            src = p.src; act = p.src2; beta = own;
            mask = beta ? 2 : 1;
        } else if (int r = pend_copy_flush(cx, st)) return r;
    }
    bool pd_zero = false;
    {
        const size_t tb = elements * sizeof(float), zb = (size_t)z * sizeof(float);
        if (mask) { EB_READS(src, tb); if (mask == 1) EB_READS(act, tb); EB_WRITES(delta, tb); } else EB_MODIFIES(delta, tb);
        EB_READS(opa, tb);
        EB_MODIFIES(gbn_g, zb); EB_MODIFIES(gbn_b, zb); EB_READS(bn_g, zb); EB_READS(variance, zb); EB_MODIFIES(mean1, zb); EB_MODIFIES(mean2, zb);
        EB_NOTES(pdelta, tb);
        if (lz_any(cx) && pdelta != delta && pdelta != opa) {
            int status = 0;
            pd_zero = lz_take(cx, st, pdelta, tb, &status);
            if (status) return status;
        }
    }
    // bytes per element: delta and opa read (and the tensor a ReLU tests), delta and the parent delta written
    ProfScope prof(cx, PROF_BN_BWD, (16.0 + (mask == 1 ? 4.0 : 0.0) + (pd_zero ? 0.0 : 4.0)) * (double)elements);
    const unsigned per = (unsigned)b * rc, S = pick_split(z, per);
    const bool vec = (rc % 4 == 0) && aligned16(delta) && aligned16(opa) && aligned16(pdelta) && aligned16(src) && (mask != 1 || aligned16(act));
    auto one = pd_zero ? (mask == 0 ? bwd_one_launch<true, 0> : mask == 1 ? bwd_one_launch<true, 1> : bwd_one_launch<true, 2>)
                       : (mask == 0 ? bwd_one_launch<false, 0> : mask == 1 ? bwd_one_launch<false, 1> : bwd_one_launch<false, 2>);
    const int r = one(dev, st, b, z, rc, vec, delta, opa, pdelta, src, act, beta, gbn_g, gbn_b, bn_g, variance, mean1, mean2);
    if (r == 0) count_launch(cx);
    if (r != kNotTaken) return r;
    float2 *partial = (float2 *)scratch(cx, (size_t)z * S * sizeof(float2));
    if (!partial) return cudaErrorMemoryAllocation;
    auto two = pd_zero ? (mask == 0 ? bwd_two_pass<true, 0> : mask == 1 ? bwd_two_pass<true, 1> : bwd_two_pass<true, 2>)
                       : (mask == 0 ? bwd_two_pass<false, 0> : mask == 1 ? bwd_two_pass<false, 1> : bwd_two_pass<false, 2>);
    two(st, S, vec, delta, opa, pdelta, src, act, beta, partial, gbn_g, gbn_b, bn_g, variance, mean1, mean2, b, z, rc);
    count_launch(cx);
    EB_LAUNCH_CHECK("gpu_batchnorm_backward");
    return 0;
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------
// BatchNorm forward for callers that are not allowed to allocate device memory.
//
// eddlb200_bn_fwd keeps its per-channel partial sums in the library's growable scratch arena,
// which it obtains with cudaMalloc the first time (and whenever a larger one is needed), and the
// device context behind it also allocates on first use.  Some hosts cannot tolerate that: a
// process whose device memory has been handed over in full to another allocator (a cudaMalloc
// from a plug-in then fails or fragments that pool), or a latency-critical loop in which the
// implicit device synchronisation of cudaMalloc / cudaFree is not acceptable.  For them this
// entry point runs the same kernels, small tensors in one launch without partial sums and the
// others with the partial sums in a fixed array that is part of the library image: kNoAllocPairs (sum, sum-of-squares) pairs = 2 MiB of device memory, held by
// every GPU that loads the library until the process exits.
//
// * It calls no cudaMalloc / cudaFree / cudaMallocHost and does not create the library's device
//   context; the caller supplies the stream.
// * The array's name is only a host-side handle.  Its device address is looked up once per
//   device with cudaGetSymbolAddress while that device is current; this happens inside the FIRST
//   call on each device, so make that first call before any stream capture begins.
// * Shapes that need more than kNoAllocPairs partial pairs (channels x slices) are rejected with
//   EDDLB200_ELIMIT.
// * All calls on a device share the one array and it keeps whatever the last call left there.
//   Nothing has to be cleared between calls: the statistics kernel overwrites every pair the
//   apply kernel reads.  Two calls that overlap on the GPU (different streams, no ordering) race
//   on the array and give wrong statistics; order them.
namespace {

constexpr unsigned kNoAllocPairs = 262144u;               // float2 pairs = 2 MiB
static __device__ __align__(256) float2 g_noalloc_partials[kNoAllocPairs];

float2 *g_noalloc_addr[EDDLB200_MAX_DEVICES] = {};
std::mutex g_noalloc_mu;

// Device address of g_noalloc_partials on `dev` (which must be current); nullptr + error text on failure.
float2 *noalloc_scratch(int dev) {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (g_noalloc_addr[dev]) return g_noalloc_addr[dev];
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_partials);
    if (e != cudaSuccess || !p) {
        cuda_status(e == cudaSuccess ? cudaErrorInvalidSymbol : e, "eddlb200_bn_fwd_noalloc(cudaGetSymbolAddress)");
        return nullptr;
    }
    g_noalloc_addr[dev] = (float2 *)p;
    return g_noalloc_addr[dev];
}

}  // namespace

extern "C" int eddlb200_bn_fwd_noalloc(int dev, int b, int z, int rc, const float *input, float *output, float *opa,
                                       float *global_mean, float *global_variance, const float *affine_g, const float *affine_b,
                                       float *mean, float *variance, int trmode, float epsilon, float momentum, float *relu_out,
                                       void *cuda_stream) {
    if (dev < 0 || dev >= EDDLB200_MAX_DEVICES) return set_error(EDDLB200_ENOINIT, "bn_fwd_noalloc: device ordinal %d out of range", dev);
    if (!(b > 0 && z > 0 && rc > 0 && input && output && global_mean && global_variance && variance) ||
        (affine_g && !(affine_b && opa)) || (trmode && !mean) || (size_t)b * rc >= 0xfffffff0u)
        return set_error(EDDLB200_EINVAL, "bn_fwd_noalloc: bad argument");
    const unsigned per = (unsigned)b * rc, S = pick_split(z, per);
    if (trmode && (size_t)z * S > kNoAllocPairs)          // inference reads no partial sums
        return set_error(EDDLB200_ELIMIT, "bn_fwd_noalloc: %d channels x %u slices need %zu partial pairs, the built-in scratch holds %u",
                         z, S, (size_t)z * S, kNoAllocPairs);
    cudaError_t e = cudaSetDevice(dev);
    if (e != cudaSuccess) return cuda_status(e, "bn_fwd_noalloc(cudaSetDevice)");
    float2 *partial = noalloc_scratch(dev);
    if (!partial) return EDDLB200_ENOINIT;
    const cudaStream_t caller = (cudaStream_t)cuda_stream;
    if (DevCtx *cx = ctx_peek(dev)) {
        // A device context exists.  It may owe deferred zeros or a recorded copy -- possibly to buffers this call never
        // sees -- and that work belongs on the library's compute stream, where whatever produces its operands runs.  It
        // is settled THERE; when the caller's stream is a different one, an event that exists since the context was
        // created is recorded behind it and the caller's stream waits on it, so the kernels below run after the settled
        // work and after everything the library had enqueued (nothing is created or allocated on this path).
        const cudaStream_t st = stream_of(cx);
        if (pend_copy_active(cx)) { if (int r = pend_copy_flush(cx, st)) return r; }
        const size_t tb = (size_t)b * z * rc * sizeof(float), zb = (size_t)z * sizeof(float);
        EB_READS(input, tb); EB_WRITES(output, tb); EB_WRITES(opa, tb); EB_WRITES(relu_out, tb);
        EB_MODIFIES(global_mean, zb); EB_MODIFIES(global_variance, zb); EB_READS(affine_g, zb); EB_READS(affine_b, zb);
        EB_MODIFIES(mean, zb); EB_MODIFIES(variance, zb);
        if (caller != st) {
            if ((e = cudaEventRecord(handoff_event(cx), st)) != cudaSuccess) return cuda_status(e, "bn_fwd_noalloc(record)");
            if ((e = cudaStreamWaitEvent(caller, handoff_event(cx), 0)) != cudaSuccess) return cuda_status(e, "bn_fwd_noalloc(wait)");
        }
    }
    const cudaStream_t st = caller;
    const bool vec = (rc % 4 == 0) && aligned16(input) && aligned16(output) && (!opa || aligned16(opa)) && (!relu_out || aligned16(relu_out));
    const Stride w = stride_of(z, rc, vec ? kBlock * 4 : kBlock);
    dim3 grid(z, S);
    if (trmode) {
        const int r = fwd_one_launch(dev, st, b, z, rc, vec, input, output, opa, global_mean, global_variance, affine_g, affine_b, mean, variance, epsilon, momentum, relu_out);
        if (r != kNotTaken) return r;
        fwd_two_pass(st, S, vec, input, output, opa, relu_out, partial, global_mean, global_variance, affine_g, affine_b, mean, variance, z, rc, per, epsilon, momentum);
    } else {
        if (vec) eb::launch(bn_fwd_apply_kernel<false, true>, grid, kBlock, 0, st, input, output, opa, relu_out, nullptr, global_mean, global_variance, affine_g, affine_b, mean, variance, per, w, epsilon, momentum);
        else eb::launch(bn_fwd_apply_kernel<false, false>, grid, kBlock, 0, st, input, output, opa, relu_out, nullptr, global_mean, global_variance, affine_g, affine_b, mean, variance, per, w, epsilon, momentum);
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_status(e, "bn_fwd_noalloc(apply)");
    return 0;
}

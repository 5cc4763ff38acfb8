// Dense-layer algebra: C = op(A)*op(B) (+C), row bias add, column/row sums.
// Replaces gpu_mult2D (cublasSgemm, EDDL src/hardware/gpu/gpu_math.cu:457-490),
// gpu_sum2D_rowwise (gpu_math.cu:517-528) and gpu_reduce_sum2D (gpu_reduction.cu:232-244,
// one atomicAdd per element); arithmetic as cpu_mult2D / cpu_sum2D_rowwise /
// cpu_reduce_sum2D (src/hardware/cpu/cpu_math.cpp:302-325,369-380; cpu_reduction.cpp:91-112).
// Three kernels share the products, each where it is the fastest (pick_route): fp32 FMA with the k slices of a tile
// meeting in cluster memory (sgemm_kernel), fp32 FMA with any number of k slices
// meeting in memory (sgemm_split_kernel), and the convolutions' tensor-core kernel.
#include <cooperative_groups.h>
#include "common.cuh"
#include "conv_common.cuh"

namespace {

using namespace eb;

constexpr int BM = 64, BN = 64, BK = 32, TB = 256;
constexpr int kMaxCluster = 8;          // portable cluster size: k slices of one output tile

// Row-major storage.  A: TA ? [k,m] : [m,k]; B: TB_ ? [n,k] : [k,n]; C: [m,n].
// The products of the nets are small (100 x 1024 x 1024): what bounds them is not arithmetic but how much of the GPU takes part
// and how long the chain load -> multiply -> combine is.  A 64 x 64 tile is computed by a CLUSTER of up to eight blocks, each
// with its own slice of k; the partial tiles meet in the blocks' shared memory, and every block adds its share of the rows from
// all of them in slice order and stores it -- one launch, no partial sums in memory.  A k step of 32 is fetched into registers
// while the one before it is multiplied (16-byte loads where VEC: rows and pointers 16-byte aligned), 4 x 4 outputs per
// thread.  A k step takes 2.45 us however few blocks there are (it is a chain of latencies): 100 x 1024 x 1024 is four of them, 13 us
// against 22 on the tensor-core kernel with its split-K and operand packing; exact fp32.
template <bool TA, bool TB_, bool VEC>
__global__ void __launch_bounds__(TB) sgemm_kernel(const float *__restrict__ A, const float *__restrict__ B, float *__restrict__ C, int inc_c,
                                                   int m, int n, int k, int k_per_slice) {
    constexpr int LD = BM + 4;
    __shared__ __align__(16) float smem[2 * BK * LD];                 // As and Bs; afterwards the 64 x 64 partial tile
    float (*As)[LD] = reinterpret_cast<float (*)[LD]>(smem), (*Bs)[LD] = reinterpret_cast<float (*)[LD]>(smem + BK * LD);
    EB_GRID_WAIT();
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int kbeg = blockIdx.z * k_per_slice, kend = min(k, kbeg + k_per_slice);
    float acc[4][4] = {};
    // An operand tile is 64 x BK = 512 pieces of four elements along the dimension that is contiguous in memory; a thread moves
    // pieces threadIdx.x and threadIdx.x + 256.  K_FAST: contiguous along k (8 pieces per row), else along the row (16 per k).
    auto fetch = [&](const float *src, bool k_fast, int rows, int row0, int ld, int k0, int piece) -> float4 {
        const int r = k_fast ? piece / (BK / 4) : (piece % 16) * 4, kk = k_fast ? (piece % (BK / 4)) * 4 : piece / 16;
        const int gr = row0 + r, gk = k0 + kk;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (k_fast) {
            if (gr < rows) {
                const float *q = src + (size_t)gr * ld + gk;
                if (VEC && gk + 4 <= kend) v = ldg4(q);
                else { if (gk < kend) v.x = __ldg(q); if (gk + 1 < kend) v.y = __ldg(q + 1); if (gk + 2 < kend) v.z = __ldg(q + 2); if (gk + 3 < kend) v.w = __ldg(q + 3); }
            }
        } else if (gk < kend) {
            const float *q = src + (size_t)gk * ld + gr;
            if (VEC && gr + 4 <= rows) v = ldg4(q);
            else { if (gr < rows) v.x = __ldg(q); if (gr + 1 < rows) v.y = __ldg(q + 1); if (gr + 2 < rows) v.z = __ldg(q + 2); if (gr + 3 < rows) v.w = __ldg(q + 3); }
        }
        return v;
    };
    auto put = [&](float (*tile)[LD], bool k_fast, int piece, float4 v) {
        if (k_fast) {
            const int r = piece / (BK / 4), kk = (piece % (BK / 4)) * 4;
            tile[kk][r] = v.x; tile[kk + 1][r] = v.y; tile[kk + 2][r] = v.z; tile[kk + 3][r] = v.w;
        } else *reinterpret_cast<float4 *>(&tile[piece / 16][(piece % 16) * 4]) = v;
    };
    float4 a0, a1, b0, b1;
    auto load = [&](int k0) {
        a0 = fetch(A, !TA, m, m0, TA ? m : k, k0, threadIdx.x); a1 = fetch(A, !TA, m, m0, TA ? m : k, k0, threadIdx.x + TB);
        b0 = fetch(B, TB_, n, n0, TB_ ? k : n, k0, threadIdx.x); b1 = fetch(B, TB_, n, n0, TB_ ? k : n, k0, threadIdx.x + TB);
    };
    load(kbeg);
    for (int k0 = kbeg; k0 < kend; k0 += BK) {
        put(As, !TA, threadIdx.x, a0); put(As, !TA, threadIdx.x + TB, a1);
        put(Bs, TB_, threadIdx.x, b0); put(Bs, TB_, threadIdx.x + TB, b1);
        __syncthreads();
        if (k0 + BK < kend) load(k0 + BK);
#pragma unroll
        for (int kk = 0; kk < BK; kk++) {
            const float4 a = *reinterpret_cast<const float4 *>(&As[kk][ty * 4]), b = *reinterpret_cast<const float4 *>(&Bs[kk][tx * 4]);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
        __syncthreads();
    }
    auto store = [&](int gm, int gn, float v) {
        float *c = C + (size_t)gm * n + gn;
        *c = inc_c == 1 ? __fadd_rn(*c, v) : (inc_c == 2 ? __fadd_rn(0.f, v) : v);          // 2: c is known to hold zeros
    };
    const unsigned slices = gridDim.z;
    if (slices == 1) {
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (m0 + ty * 4 + i < m && n0 + tx * 4 + j < n) store(m0 + ty * 4 + i, n0 + tx * 4 + j, acc[i][j]);
        return;
    }
    static_assert(BM * BN <= 2 * BK * LD, "the partial tile takes the place of the operand tiles");
#pragma unroll
    for (int i = 0; i < 4; i++) *reinterpret_cast<float4 *>(smem + (ty * 4 + i) * BN + tx * 4) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    cluster.sync();
    const float *peer[kMaxCluster];
    for (unsigned z = 0; z < kMaxCluster; z++) peer[z] = cluster.map_shared_rank(smem, z < slices ? z : 0);
    for (int e = (int)blockIdx.z * TB + threadIdx.x; e < BM * BN; e += (int)slices * TB) {
        float v[kMaxCluster];
#pragma unroll
        for (unsigned z = 0; z < kMaxCluster; z++) v[z] = z < slices ? peer[z][e] : 0.f;
        float s = v[0];
#pragma unroll
        for (unsigned z = 1; z < kMaxCluster; z++) if (z < slices) s = __fadd_rn(s, v[z]);
        const int gm = m0 + e / BN, gn = n0 + e % BN;
        if (gm < m && gn < n) store(gm, gn, s);
    }
    cluster.sync();                     // a block's shared memory outlives the reads of the others
}

template <bool TA, bool TB_, bool VEC>
int launch_sgemm(DevCtx *cx, cudaStream_t st, const float *a, const float *b, float *c, int inc_c, int m, int n, int k, int slices, int kps) {
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension; at[1].val.clusterDim.x = 1; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = slices;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((n + BN - 1) / BN, (m + BM - 1) / BM, slices); cfg.blockDim = dim3(TB); cfg.stream = st; cfg.attrs = at; cfg.numAttrs = 2;
    cudaLaunchKernelEx(&cfg, sgemm_kernel<TA, TB_, VEC>, a, b, c, inc_c, m, n, k, kps);
    EB_LAUNCH_CHECK("gpu_mult2D");
    return 0;
}

// The same tile with any number of k slices, which leave partial tiles in memory (part; null = one slice, straight into C).  For
// reductions that eight slices do not make short (8 x 2 x 100000: 70 us, 615 with eight), and, with half the step, for
// outer products of up to 16 terms, where sgemm_kernel's step of 32 is mostly padding (4096 x 4096 x 1: 45 us against 60).
constexpr int SBK = 16;
__global__ void __launch_bounds__(TB) sgemm_split_kernel(const float *__restrict__ A, int ta, const float *__restrict__ B, int tb,
                                                         float *__restrict__ C, int inc_c, int m, int n, int k, int k_per_split,
                                                         float *__restrict__ part) {
    EB_GRID_WAIT();
    __shared__ float As[SBK][BM + 4];
    __shared__ float Bs[SBK][BN + 4];
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float acc[4][4] = {};
    const int kbeg = blockIdx.z * k_per_split;
    int kend = k;
    if (part) { kend = min(k, kbeg + k_per_split); C = part + (size_t)blockIdx.z * m * n; inc_c = 0; }
    for (int k0 = kbeg; k0 < kend; k0 += SBK) {
        for (int e = threadIdx.x; e < BM * SBK; e += TB) {
            // choose the traversal that is contiguous in memory
            int mi, ki;
            if (ta) { mi = e % BM; ki = e / BM; } else { ki = e % SBK; mi = e / SBK; }
            const int gm = m0 + mi, gk = k0 + ki;
            float v = 0.f;
            if (gm < m && gk < kend) v = ta ? A[(size_t)gk * m + gm] : A[(size_t)gm * k + gk];
            As[ki][mi] = v;
        }
        for (int e = threadIdx.x; e < BN * SBK; e += TB) {
            int ni, ki;
            if (tb) { ki = e % SBK; ni = e / SBK; } else { ni = e % BN; ki = e / BN; }
            const int gn = n0 + ni, gk = k0 + ki;
            float v = 0.f;
            if (gn < n && gk < kend) v = tb ? B[(size_t)gn * k + gk] : B[(size_t)gk * n + gn];
            Bs[ki][ni] = v;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < SBK; kk++) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; i++) a[i] = As[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; j++) b[j] = Bs[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int gm = m0 + ty * 4 + i;
        if (gm >= m) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int gn = n0 + tx * 4 + j;
            if (gn >= n) continue;
            float *c = C + (size_t)gm * n + gn;
            *c = inc_c == 1 ? __fadd_rn(*c, acc[i][j]) : (inc_c == 2 ? __fadd_rn(0.f, acc[i][j]) : acc[i][j]);     // 2: c is known to hold zeros
        }
    }
}

// c[i] = (inc_c ? c[i] : 0) + part[0][i] + part[1][i] + ...   (fixed order)
__global__ void __launch_bounds__(256) sgemm_combine_kernel(const float *__restrict__ part, float *__restrict__ c, size_t count, int splits, int inc_c) {
    EB_GRID_WAIT();
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += stride) {
        float v = inc_c ? c[i] : 0.f;
        for (int z = 0; z < splits; z++) v = __fadd_rn(v, part[(size_t)z * count + i]);
        c[i] = v;
    }
}

int launch_split(DevCtx *cx, cudaStream_t st, const float *a, int ta, const float *b, int tb, float *c, int inc_c, int m, int n, int k, int splits, int kps) {
    dim3 grid((n + BN - 1) / BN, (m + BM - 1) / BM, splits);
    const size_t count = (size_t)m * n;
    float *part = splits > 1 ? (float *)scratch(cx, count * splits * sizeof(float)) : nullptr;
    if (!part) grid.z = splits = 1, kps = k;               // no room for partial tiles: unsplit, straight into C
    eb::launch(sgemm_split_kernel, grid, TB, 0, st, a, ta, b, tb, c, inc_c, m, n, k, kps, part);
    EB_LAUNCH_CHECK("gpu_mult2D");
    if (splits == 1) return 0;
    eb::launch(sgemm_combine_kernel, grid_for(count, 256), 256, 0, st, part, c, count, splits, inc_c == 1);
    EB_LAUNCH_CHECK("gpu_mult2D(combine)");
    return 0;
}

// Which kernel runs a product.  The estimates (microseconds) are fits to 420 products of m, n and k between 1 and 100000, plain and
// transposed, warm and with a flushed L2; over these the choice takes 10.9 ms where the best kernel for each would take 10.8,
// the cluster kernel alone 19.6 and the other two alone 14.0.
enum class Route { Cluster, Split, TensorCore };
struct GemmPlan { Route route; int slices, kps; };
GemmPlan pick_route(int m, int n, int k, bool ta, bool tc_allowed) {
    const double mnk = (double)m * n * k;
    const long long tiles = (long long)((n + BN - 1) / BN) * ((m + BM - 1) / BM);
    // cluster kernel: two blocks per SM where the tiles alone do not give them, slices of at least 64 (two k steps)
    int slices = 1;
    while (slices < kMaxCluster && tiles * slices * 2 <= 2 * EDDLB200_NUM_SMS && k >= slices * 2 * 64) slices *= 2;
    const int kps = ((k + slices - 1) / slices + BK - 1) / BK * BK, steps = kps / BK;
    const GemmPlan cluster{Route::Cluster, slices, kps};
    // split kernel: as many slices of at least 64 as give two blocks per SM
    int splits = 1;
    if (tiles < EDDLB200_NUM_SMS) {
        splits = (int)((2 * EDDLB200_NUM_SMS + tiles - 1) / tiles);
        if (splits > k / 64) splits = k / 64;
        if (splits < 1) splits = 1;
    }
    const int skps = splits == 1 ? k : ((k + splits - 1) / splits + SBK - 1) / SBK * SBK;
    if (splits > 1) splits = (k + skps - 1) / skps;
    const GemmPlan split{Route::Split, splits, skps};
    const bool tc = tc_allowed && k >= 32 && mnk >= 67108864.0;
    // From 2^29 multiply-adds on (whatever the shape) the tensor cores win.
    if (tc && mnk >= 536870912.0) return GemmPlan{Route::TensorCore, 1, k};
    // Outer products: the stores count once there is more than a wave of tiles, the launch and the latency before that.
    if (k <= SBK) return tiles <= 2 * EDDLB200_NUM_SMS ? cluster : split;
    if (steps <= 4) return cluster;
    const double waves = (double)tiles * slices / EDDLB200_NUM_SMS, cluster_us = 2.5 + steps * (1.3 * waves > 2.45 ? 1.3 * waves : 2.45);
    double other_us;
    if (tc) {
        // the packing and the gather of a row-major A (not transposed: lanes run along m) grow with the rows of the first 128-row tile
        const double rows = (m < 128 ? m : 128) / 128.0;
        other_us = conv_tc_gemm_us(m, n, k) + (ta ? 10.0 * rows : 3.0 + 14.0 * rows) + 8.0 * m * (double)n / 5.0e6;
    } else {
        const double over = (double)tiles * splits / (2 * EDDLB200_NUM_SMS);
        other_us = 5.0 + 2.65 * ((skps + SBK - 1) / SBK) * (over > 1.0 ? over : 1.0) + (splits > 1 ? 3.0 + 0.07 * splits : 0.0);
    }
    if (cluster_us <= 1.1 * other_us) return cluster;
    return tc ? GemmPlan{Route::TensorCore, 1, k} : split;
}

__global__ void __launch_bounds__(256) rowbias_kernel(const float *__restrict__ a, const float *__restrict__ b, float *__restrict__ c, size_t total, int cols) {
    EB_GRID_WAIT();
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x; p < total; p += stride)
        c[p] = __fadd_rn(a[p], __ldg(b + (total < (size_t(1) << 32) ? (unsigned)p % (unsigned)cols : p % cols)));
}

// axis 0: one thread per column walks the rows in order (the reference's order), coalesced
// across columns.  axis 1: one warp per row.
__global__ void __launch_bounds__(256) colsum_kernel(const float *__restrict__ a, float *__restrict__ b, int rows, int cols, int inc_b) {
    EB_GRID_WAIT();
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= cols) return;
    float s = inc_b ? b[j] : 0.f;
    int i = 0;
    for (; i + 16 <= rows; i += 16) {               // sixteen loads in flight, added in order: one memory latency per sixteen rows
        float v[16];
#pragma unroll
        for (int r = 0; r < 16; r++) v[r] = __ldg(a + (size_t)(i + r) * cols + j);
#pragma unroll
        for (int r = 0; r < 16; r++) s = __fadd_rn(s, v[r]);
    }
    for (; i < rows; i++) s = __fadd_rn(s, __ldg(a + (size_t)i * cols + j));
    b[j] = s;
}
__global__ void __launch_bounds__(256) rowsum_kernel(const float *__restrict__ a, float *__restrict__ b, int rows, int cols, int inc_b) {
    EB_GRID_WAIT();
    const int lane = threadIdx.x & 31;
    const int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (r >= rows) return;
    float s = 0.f;
    for (int j = lane; j < cols; j += 32) s += a[(size_t)r * cols + j];
    s = warp_sum(s);
    if (lane == 0) b[r] = inc_b ? __fadd_rn(b[r], s) : s;
}

}  // namespace

using namespace eb;

extern "C" {

int eddlb200_mult2d(int dev, const float *a, int ta, const float *b, int tb, float *c, int inc_c, int m, int n, int k) {
    EB_CTX(dev);
    EB_REQUIRE(a && b && c && m >= 0 && n >= 0 && k >= 0, "gpu_mult2D");
    if (m == 0 || n == 0) return 0;
    EB_READS(a, (size_t)m * k * sizeof(float)); EB_READS(b, (size_t)k * n * sizeof(float));
    if (inc_c && lz_any(cx) && c != a && c != b) {
        int status = 0;
        if (lz_take(cx, st, c, (size_t)m * n * sizeof(float), &status)) inc_c = 2;
        if (status) return status;
    }
    if (inc_c == 1) EB_MODIFIES(c, (size_t)m * n * sizeof(float)); else EB_WRITES(c, (size_t)m * n * sizeof(float));
    ProfScope prof(cx, PROF_GEMM, 2.0 * m * (double)n * k);
    GemmPlan plan = pick_route(m, n, k, ta != 0, conv_tc_allowed());          // a library forced to the FMA path stays on the FMA kernels
    if (plan.route == Route::TensorCore) {
        const int r = conv_tc_gemm(cx, st, a, ta, b, tb, c, inc_c, m, n, k, 0);
        if (r != kNotTaken) return r;
        plan = pick_route(m, n, k, ta != 0, false);
    }
    if (plan.route == Route::Split) return launch_split(cx, st, a, ta, b, tb, c, inc_c, m, n, k, plan.slices, plan.kps);
    const int slices = plan.slices, kps = plan.kps;
    const bool vec = aligned16(a) && aligned16(b) && (ta ? m : k) % 4 == 0 && (tb ? k : n) % 4 == 0;
    if (ta) {
        if (tb) return vec ? launch_sgemm<true, true, true>(cx, st, a, b, c, inc_c, m, n, k, slices, kps) : launch_sgemm<true, true, false>(cx, st, a, b, c, inc_c, m, n, k, slices, kps);
        return vec ? launch_sgemm<true, false, true>(cx, st, a, b, c, inc_c, m, n, k, slices, kps) : launch_sgemm<true, false, false>(cx, st, a, b, c, inc_c, m, n, k, slices, kps);
    }
    if (tb) return vec ? launch_sgemm<false, true, true>(cx, st, a, b, c, inc_c, m, n, k, slices, kps) : launch_sgemm<false, true, false>(cx, st, a, b, c, inc_c, m, n, k, slices, kps);
    return vec ? launch_sgemm<false, false, true>(cx, st, a, b, c, inc_c, m, n, k, slices, kps) : launch_sgemm<false, false, false>(cx, st, a, b, c, inc_c, m, n, k, slices, kps);
}

int eddlb200_sum2d_rowwise(int dev, const float *a, const float *b, float *c, int rows, int cols) {
    EB_CTX(dev);
    EB_REQUIRE(a && b && c && rows >= 0 && cols >= 0, "gpu_sum2D_rowwise");
    const size_t total = (size_t)rows * cols;
    if (!total) return 0;
    EB_READS(a, total * sizeof(float)); EB_READS(b, (size_t)cols * sizeof(float));
    if (c != a) EB_WRITES(c, total * sizeof(float));
    eb::launch(rowbias_kernel, grid_for(total, 256), 256, 0, st, a, b, c, total, cols);
    EB_LAUNCH_CHECK("gpu_sum2D_rowwise");
    return 0;
}

int eddlb200_reduce_sum2d(int dev, const float *a, float *b, int rows, int cols, int axis, int inc_b) {
    EB_CTX(dev);
    EB_REQUIRE(a && b && rows >= 0 && cols >= 0 && (axis == 0 || axis == 1), "gpu_reduce_sum2D");
    EB_READS(a, (size_t)rows * cols * sizeof(float));
    if (inc_b) EB_MODIFIES(b, (size_t)(axis == 0 ? cols : rows) * sizeof(float)); else EB_WRITES(b, (size_t)(axis == 0 ? cols : rows) * sizeof(float));
    if (axis == 0) {
        if (!cols) return 0;
        eb::launch(colsum_kernel, (cols + 63) / 64, 64, 0, st, a, b, rows, cols, inc_b);
    } else {
        if (!rows) return 0;
        eb::launch(rowsum_kernel, (rows + 7) / 8, 256, 0, st, a, b, rows, cols, inc_b);
    }
    EB_LAUNCH_CHECK("gpu_reduce_sum2D");
    return 0;
}

}  // extern "C"

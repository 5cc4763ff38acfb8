// Backward-weight of Conv2D on pairs of CTAs (tcgen05.mma, cta_group::2): gw[n][m] = sum over pixels of A[m][pixel] B[n][pixel].
//
// Both operands run along the pixels of NCHW planes, so TMA delivers them as K-major tiles of 32 pixels.  What bounds such a kernel is
// shared-memory bandwidth (128 bytes per SM and cycle).  Bytes moved per K-block of a 128 x 128 tile in 3xTF32 (12 MMAs, 768 cycles):
//                                  1x1 one CTA   1x1 pair    3x3 one CTA   3x3 pair
//     landing of x and dy             32 KB        24 KB         26 KB       17.5 KB
//     conversion (read, write)        64 KB        48 KB         80 KB        64 KB
//     operand reads of the MMAs       96 KB        72 KB         96 KB        72 KB
//     cycles                          1536         1152          1616         1228
// A pair computes 256 rows with M = 256 instructions; each CTA lands, converts and holds its own 128 rows of A and HALF of B.
// The counts are upper bounds; measured with fill and drain: 1172 cycles (3x3 pair, tensor pipe busy 65 %) and 1067 (1x1 pair, 70 %),
// profiles/conv_pairs_bn_gemm.md.
// Whole calls, single launches behind a flushed L2, 3xTF32, igemm_tc_kernel on the same layer -> this kernel: 64 x 256 x 56 x 56, 256
// filters, 3x3: 1574 -> 1181 us; 64 x 128 x 28 x 28, 3x3: 126 -> 93; 64 x 256 x 14 x 14, 3x3: 142 -> 106; 64 x 1024 x 14 x 14, 256
// filters, 1x1: 52 -> 44; 64 x 512 x 28 x 28, 256 filters, 1x1: 81 -> 67.  With one lane per pixel and 4-byte accesses in the SLAB
// producers the first of these took 1516 us: four times the shared-memory instructions for the same bytes.
//
// SLAB = false, 1x1 stride-1 unpadded layers: A rows are the channels of x or, swapped, the filters of dy -- whichever fills 256
// rows better -- and the landed values are the hi planes as they are.  SLAB = true, 3x3 stride-1 "same" layers: the 128 rows of a
// CTA are the nine taps of 14 channels (two rows stay zero), built from one raw slab per K-block; B is dy.
//
//   warps 0-7    producers: two groups of four warps take alternate K-blocks; they write the lo planes (SLAB: all of A)
//   warp  8      (first CTA of the pair) one lane issues the MMAs
//   warp  9      one lane keeps the landing ring of its CTA filled by TMA
//   warps 10-17  epilogue: two warps per TMEM lane quarter, half of the columns each
// What lands lives in a ring of HI slots, what the producers write in a ring of three LO slots: with two, a group could convert only
// while the other group's K-block was being multiplied.  Every wait is bounded as in igemm_tc_kernel.
#pragma once
#include "tc_ptx.cuh"

namespace {

using namespace eb;

// a tile's 126 rows of the slab-fed kernels (this one and igemm_tc_kernel's TMA = 4): the nine taps of 14 channels, the last two rows
// of the 128 stay zero.  A K-block is 32 pixels of one image; one slab of [16 channels][152 pixels] -- the 32 pixels plus a halo
// of W + 1 either side, its start rounded down to 16 bytes -- serves all rows (W <= 57)
constexpr int WS_CH = 14, WS_ROWS = 9 * WS_CH, WS_SLAB_PX = 152, WS_SLAB_CH = 16;

constexpr int WG_THREADS = 18 * 32;

struct WgParams {
    CUtensorMap mapA, mapB;                  // boxes: A [128 channels or 16 slab channels][32 or 152 pixels], B [BN / 2][32 pixels]
    float *out;                              // element (m, n) at m * m_stride + n * n_stride
    int *status;
    long long split_stride, m_stride, n_stride;
    int M_total, N_total, tiles_m, tiles_n, splits, kblocks, kblocks_per_split;     // tiles_m: of 256 rows (SLAB: 252)
    int chunks_per_image, img_w, plane_px, nmain, accumulate, raw_hi;
};

template <int BN_, bool SPLIT3, bool SLAB>
struct WgLayout {
    static constexpr int A_BYTES = BM * BK * 4, BH_BYTES = BN_ / 2 * BK * 4;
    static constexpr int X_BYTES = SLAB ? WS_SLAB_CH * WS_SLAB_PX * 4 : A_BYTES;
    static constexpr int LO_BYTES = (SLAB ? A_BYTES : 0) + (SPLIT3 ? A_BYTES + BH_BYTES : 0);
    static constexpr int LO_SLOTS = 3;
    static constexpr int BAR_BYTES = 512, BUDGET = 232448 - 1024 - BAR_BYTES - LO_SLOTS * LO_BYTES;
    static constexpr int HI_SLOTS = BUDGET / (BH_BYTES + X_BYTES) > 8 ? 8 : BUDGET / (BH_BYTES + X_BYTES);
    static_assert(HI_SLOTS >= 4, "a copy takes about two K-blocks to land");
    static_assert((2 * LO_SLOTS + 2 * HI_SLOTS + 4) * 8 + 16 <= BAR_BYTES, "barrier words");
    static constexpr int SMEM_BYTES = 1024 + HI_SLOTS * (BH_BYTES + X_BYTES) + LO_SLOTS * LO_BYTES + BAR_BYTES;
};

template <int BN_, bool SPLIT3, bool SLAB>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(WG_THREADS, 1) conv_wg_kernel(const __grid_constant__ WgParams P) {
    using L = WgLayout<BN_, SPLIT3, SLAB>;
    constexpr int HS = L::HI_SLOTS, LS = L::LO_SLOTS;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *hib = smem, *lo_base = smem + HS * L::BH_BYTES, *x_base = lo_base + LS * L::LO_BYTES;      // swizzled tiles on 1024 bytes, slabs on 128
    uint64_t *bars = (uint64_t *)(x_base + HS * L::X_BYTES);
    uint32_t *tmem_slot = (uint32_t *)(bars + 2 * LS + 2 * HS + 4);
    volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
    const uint32_t bar_full = smem_u32(bars), bar_empty = bar_full + 8 * LS, bar_landed = bar_empty + 8 * LS, bar_hi_empty = bar_landed + 8 * HS;
    const uint32_t bar_acc_full = bar_hi_empty + 8 * HS, bar_acc_empty = bar_acc_full + 16;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = (int)cluster_rank(), pair = (int)(blockIdx.x >> 1), pairs = (int)(gridDim.x >> 1);
    const int tiles_mn = P.tiles_m * P.tiles_n, total_tiles = tiles_mn * P.splits;
    const int nacc = P.nmain + (SPLIT3 ? 1 : 0), set_cols = nacc * BN_, nsets = 512 / set_cols >= 2 ? 2 : 1;
    constexpr int CTA_ROWS = SLAB ? WS_ROWS : BM;

    if (tid == 0) {
        for (int s = 0; s < LS; s++) { mbar_init(bar_full + 8 * s, 8); mbar_init(bar_empty + 8 * s, 1); }           // four warps of each CTA
        for (int s = 0; s < HS; s++) { mbar_init(bar_landed + 8 * s, 1); mbar_init(bar_hi_empty + 8 * s, 1); }
        for (int s = 0; s < 2; s++) { mbar_init(bar_acc_full + 8 * s, 1); mbar_init(bar_acc_empty + 8 * s, 16); }   // eight warps of each CTA
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8) tmem_alloc_pair(smem_u32(tmem_slot), 512);
    if constexpr (SLAB) {                                    // the two rows of A that hold nothing
        constexpr int PLANES = SPLIT3 ? 2 : 1;
        if (tid < LS * PLANES * 16) {
            uint8_t *plane = lo_base + tid / (PLANES * 16) * L::LO_BYTES + tid / 16 % PLANES * L::A_BYTES;
            *(float4 *)(plane + WS_ROWS * 128 + (tid & 15) * 16) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        fence_async_smem();
    }
    EB_GRID_WAIT();
    tc_fence_before();
    __syncthreads();
    cluster_arrive(); cluster_wait();                        // the other CTA's barriers are initialised before anything arrives on them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    bool failed = false;
    int fail_code = 0;

    auto kb_range = [&](int t, int &kb0, int &nkb) {
        kb0 = (t / tiles_mn) * P.kblocks_per_split;
        nkb = min(P.kblocks, kb0 + P.kblocks_per_split) - kb0;
    };

    if (warp < 8) {
        // ============================ producers ============================
        const int group = warp >> 2, wq = warp & 3, gtid = tid & 127;
        const uint32_t full_of_first = map_to_rank(bar_full, 0);
        // the K-blocks of the CTA's sequence that belong to this group
        int t = pair, kb0 = 0, nkb = 0, it = group;
        auto settle = [&]() {
            while (t < total_tiles) {
                kb_range(t, kb0, nkb);
                if (it < nkb) return;
                it -= nkb; t += pairs;
            }
        };
        // lo = v - hi; all of a plane's loads go out before its first store (the compiler cannot move a shared-memory load above an
        // earlier shared-memory store)
        auto split_plane = [&](uint8_t *hi_plane, uint8_t *lo_plane, auto bytes_c) {
            constexpr int BYTES = decltype(bytes_c)::value, PIECES = BYTES / (128 * 16);
            static_assert(PIECES * 128 * 16 == BYTES, "whole pieces");
            float4 v[PIECES];
#pragma unroll
            for (int i = 0; i < PIECES; i++) v[i] = *(const float4 *)(hi_plane + (gtid + 128 * i) * 16);
#pragma unroll
            for (int i = 0; i < PIECES; i++) {
                float4 hi, lo;
                split_tf32(v[i].x, hi.x, lo.x); split_tf32(v[i].y, hi.y, lo.y); split_tf32(v[i].z, hi.z, lo.z); split_tf32(v[i].w, hi.w, lo.w);
                *(float4 *)(lo_plane + (gtid + 128 * i) * 16) = lo;
                if (!P.raw_hi) *(float4 *)(hi_plane + (gtid + 128 * i) * 16) = hi;
            }
        };
        // SLAB: a quarter warp writes whole 128-byte rows, each thread 16 bytes = four pixels.  For one channel and one row of the filter it
        // reads the six slab elements that the three horizontal taps of its pixels see (as aligned 16-byte loads, shifted in registers)
        // and stores three rows of A.  The 14 channels x 3 filter rows are dealt to the group's sixteen quarter warps.
        constexpr int JOBS = 3 * WS_CH, ROUNDS = (JOBS + 15) / 16;
        const int chunk = lane & 7;
        int job_src[SLAB ? ROUNDS : 1], job_row[SLAB ? ROUNDS : 1];          // row -1: no job
        if constexpr (SLAB) {
#pragma unroll
            for (int i = 0; i < ROUNDS; i++) {
                const int job = 16 * i + 4 * wq + (lane >> 3), c = job / 3, tr = job - 3 * c;
                job_src[i] = job < JOBS ? c * WS_SLAB_PX + tr * P.img_w + 4 * chunk : 0;
                job_row[i] = job < JOBS ? 3 * job : -1;                      // row 9 c + 3 tr
            }
        }
        settle();
        for (int g = group; t < total_tiles; g += 2) {
            const int h = g % HS, l = g % LS;
            if (!mbar_wait_warp(bar_landed + 8 * h, (g / HS) & 1, abort_flag)) { failed = true, fail_code = 1; break; }
            if (!mbar_wait_warp(bar_empty + 8 * l, ((g / LS) & 1) ^ 1, abort_flag)) { failed = true, fail_code = 2; break; }
            uint8_t *lo_slot = lo_base + l * L::LO_BYTES;
            if constexpr (SLAB) {
                const int W = P.img_w, x0 = ((kb0 + it) % P.chunks_per_image) * 32, first = x0 - W - 1;
                const int base = ((first + 4096) & ~3) - 4096, px = x0 + 4 * chunk;
                int q = px % W;
                // bit i: pixel i has a left / right neighbour in its image row (planes are a multiple of four pixels: all four or none exist)
                const bool inside = px < P.plane_px;
                uint32_t left = 0, right = 0;
#pragma unroll
                for (int i = 0; i < 4; i++) { left |= inside && q != 0 ? 1u << i : 0u; right |= inside && q != W - 1 ? 1u << i : 0u; q = q + 1 == W ? 0 : q + 1; }
                const float *slab = (const float *)(x_base + h * L::X_BYTES);
                float4 f[ROUNDS][3];
#pragma unroll
                for (int r = 0; r < ROUNDS; r++) {
                    const float4 *src = (const float4 *)(slab + ((job_src[r] + first - base) & ~3));
                    f[r][0] = src[0]; f[r][1] = src[1]; f[r][2] = src[2];
                }
#pragma unroll
                for (int r = 0; r < ROUNDS; r++) {
                    if (job_row[r] < 0) continue;
                    const int shift = (job_src[r] + first - base) & 3;
                    const float e[9] = {f[r][0].x, f[r][0].y, f[r][0].z, f[r][0].w, f[r][1].x, f[r][1].y, f[r][1].z, f[r][1].w, f[r][2].x};
                    float u[7], v[6];
#pragma unroll
                    for (int i = 0; i < 7; i++) u[i] = shift & 2 ? e[i + 2] : e[i];
#pragma unroll
                    for (int i = 0; i < 6; i++) v[i] = shift & 1 ? u[i + 1] : u[i];
#pragma unroll
                    for (int ts = 0; ts < 3; ts++) {
                        const uint32_t keep = ts == 0 ? left : ts == 2 ? right : inside ? 15u : 0u;
                        const int row = job_row[r] + ts;
                        const uint32_t o = swz_chunk(row, chunk);
                        const float4 w = make_float4(keep & 1u ? v[ts] : 0.f, keep & 2u ? v[ts + 1] : 0.f, keep & 4u ? v[ts + 2] : 0.f, keep & 8u ? v[ts + 3] : 0.f);
                        if (SPLIT3) {
                            float4 hi, lo;
                            split_tf32(w.x, hi.x, lo.x); split_tf32(w.y, hi.y, lo.y); split_tf32(w.z, hi.z, lo.z); split_tf32(w.w, hi.w, lo.w);
                            *(float4 *)(lo_slot + o) = hi; *(float4 *)(lo_slot + L::A_BYTES + o) = lo;
                        } else *(float4 *)(lo_slot + o) = w;
                    }
                }
                if constexpr (SPLIT3) split_plane(hib + h * L::BH_BYTES, lo_slot + 2 * L::A_BYTES, std::integral_constant<int, L::BH_BYTES>{});
            } else if constexpr (SPLIT3) {
                split_plane(x_base + h * L::X_BYTES, lo_slot, std::integral_constant<int, L::A_BYTES>{});
                split_plane(hib + h * L::BH_BYTES, lo_slot + L::A_BYTES, std::integral_constant<int, L::BH_BYTES>{});
            }
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(full_of_first + 8 * l);
            it += 2; settle();
        }
    } else if (warp == 8) {
        // ============================ MMA issuer (one lane of the first CTA), as in igemm_tc_kernel ============================
        if (rank == 0 && elect_one()) {
            constexpr uint32_t idesc = make_idesc_pair(BN_);
            constexpr uint32_t DESC_HI = 64u | (1u << 14) | (2u << 29);            // upper word of make_desc()
            auto desc = [&](uint32_t lo) { return ((uint64_t)DESC_HI << 32) | lo; };
            auto lo_word = [&](const uint8_t *p) { return ((smem_u32(p) >> 4) & 0x3FFFu) | (1u << 16); };
            const uint32_t hib_lo = lo_word(hib), lo_lo = lo_word(lo_base), x_lo = lo_word(x_base);
            constexpr uint32_t A_STEP = (uint32_t)L::A_BYTES >> 4, B_STEP = (uint32_t)L::BH_BYTES >> 4, LO_STEP = (uint32_t)L::LO_BYTES >> 4;
            const int nmain = P.nmain;
            const uint32_t rot_step = nmain > 1 ? (uint32_t)BN_ : 0u;
            uint32_t s = 0, phase = 0, wh = 0, ready = 0, set_phase = 1;
            int set = 0;
            for (int t = pair; t < total_tiles && !failed; t += pairs) {
                int kb0, nkb; kb_range(t, kb0, nkb);
                if (!mbar_wait(bar_acc_empty + 8 * set, set_phase, abort_flag)) { failed = true, fail_code = 3; break; }
                tc_fence_after();
                uint32_t d0 = tmem_base + (uint32_t)(set * set_cols), d1 = d0 + rot_step, d2 = d1 + rot_step;
                const uint32_t d_small = d0 + (uint32_t)(nmain * BN_);
                for (int it = 0; it < nkb; it++) {
                    if (!ready && !mbar_wait(bar_full + 8 * s, phase, abort_flag)) { failed = true, fail_code = 4; break; }
                    tc_fence_after();
                    const uint32_t next_s = s + 1 == LS ? 0u : s + 1, next_phase = phase ^ (s + 1 == LS ? 1u : 0u);
                    const uint32_t slot = lo_lo + s * LO_STEP, b_hi = hib_lo + wh * B_STEP;
                    const uint32_t a_hi = SLAB ? slot : x_lo + wh * A_STEP, a_lo = SLAB ? slot + A_STEP : slot, b_lo = a_lo + A_STEP;
                    const uint32_t old0 = it ? 1u : 0u, old12 = it || nmain == 1 ? 1u : 0u;        // an accumulator's first k-step overwrites it
#pragma unroll
                    for (int ks = 0; ks < BK / 8; ks++) {
                        const uint32_t o = 2u * ks;
                        if (SPLIT3) {
                            umma_tf32_pair(d_small, desc(a_lo + o), desc(b_hi + o), idesc, ks ? 1u : old0);
                            umma_tf32_pair(d_small, desc(a_hi + o), desc(b_lo + o), idesc, 1u);
                        }
                        umma_tf32_pair(ks == 1 ? d1 : ks == 2 ? d2 : d0, desc(a_hi + o), desc(b_hi + o), idesc, ks == 0 ? old0 : ks == 3 ? 1u : old12);
                        if (ks == 1) ready = mbar_test(bar_full + 8 * next_s, next_phase);
                    }
                    const uint32_t was0 = d0;
                    d0 = d1; d1 = d2; d2 = was0;
                    umma_commit_pair(bar_empty + 8 * s);
                    umma_commit_pair(bar_hi_empty + 8 * wh);
                    s = next_s; phase = next_phase;
                    if (++wh == HS) wh = 0;
                }
                if (failed) break;
                umma_commit_pair(bar_acc_full + 8 * set);
                if (++set == nsets) { set = 0; set_phase ^= 1u; }
            }
        }
        __syncwarp();
    } else if (warp == 9) {
        // ============================ TMA (one lane of each CTA) ============================
        if (lane == 0) {
            int g = 0;
            for (int t = pair; t < total_tiles && !failed; t += pairs) {
                int kb0, nkb; kb_range(t, kb0, nkb);
                const int mn = t % tiles_mn, m0 = (2 * (mn % P.tiles_m) + rank) * (SLAB ? WS_CH : BM), n0 = (mn / P.tiles_m) * BN_ + rank * (BN_ / 2);
                int img = kb0 / P.chunks_per_image, chunk = kb0 % P.chunks_per_image;
                for (int it = 0; it < nkb; it++, g++) {
                    const int h = g % HS;
                    if (!mbar_wait(bar_hi_empty + 8 * h, ((g / HS) & 1) ^ 1, abort_flag)) { failed = true, fail_code = 5; break; }
                    const int x0 = chunk * 32, xa = SLAB ? ((x0 - P.img_w - 1 + 4096) & ~3) - 4096 : x0;
                    mbar_expect_tx(bar_landed + 8 * h, (uint32_t)(L::BH_BYTES + L::X_BYTES));
                    tma_load_3d(smem_u32(hib + h * L::BH_BYTES), &P.mapB, x0, n0, img, bar_landed + 8 * h);
                    tma_load_3d(smem_u32(x_base + h * L::X_BYTES), &P.mapA, xa, m0, img, bar_landed + 8 * h);
                    if (++chunk == P.chunks_per_image) { chunk = 0; img++; }
                }
            }
            // the last arrivals on this CTA's ring barriers come from the first CTA's MMA issuer: stay until they are in
            for (int i = 0; i < HS && i < g && !failed; i++) {
                const int k = g - 1 - i;
                if (!mbar_wait(bar_hi_empty + 8 * (k % HS), (k / HS) & 1, abort_flag)) { failed = true, fail_code = 6; }
                if (i < LS && !failed && !mbar_wait(bar_empty + 8 * (k % LS), (k / LS) & 1, abort_flag)) { failed = true, fail_code = 6; }
            }
        }
        __syncwarp();
    } else {
        // ============================ epilogue (warps 10-17) ============================
        const int quarter = warp & 3, half = (warp - 10) >> 2;
        constexpr int COLS = BN_ >= 64 ? BN_ / 2 : 32, NC = COLS / 32;          // BN = 32: the second half has nothing to drain
        const uint32_t empty_of_first = map_to_rank(bar_acc_empty, 0);
        int set = 0; uint32_t set_phase = 0;
        for (int t = pair; t < total_tiles; t += pairs) {
            if (!mbar_wait_warp(bar_acc_full + 8 * set, set_phase, abort_flag)) { failed = true, fail_code = 7; break; }
            tc_fence_after();
            const bool idle = BN_ < 64 && half == 1;
            float acc[NC][32];
            const uint32_t base = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(set * set_cols + half * COLS);
            if (!idle) {
#pragma unroll
                for (int c = 0; c < 2 * NC; c++) {              // sixteen columns at a time: the sums of all columns stay in registers
                    uint32_t r[16];
                    tmem_ld16(base + c * 16, r);
#pragma unroll
                    for (int j = 0; j < 16; j++) acc[c / 2][(c & 1) * 16 + j] = __uint_as_float(r[j]);
#pragma unroll 1
                    for (int a = 1; a < nacc; a++) {
                        tmem_ld16(base + (uint32_t)(a * BN_ + c * 16), r);
#pragma unroll
                        for (int j = 0; j < 16; j++) acc[c / 2][(c & 1) * 16 + j] = __fadd_rn(acc[c / 2][(c & 1) * 16 + j], __uint_as_float(r[j]));
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(empty_of_first + 8 * set);
            if (++set == nsets) { set = 0; set_phase ^= 1u; }
            if (idle) continue;
            const int mn = t % tiles_mn, row = quarter * 32 + lane, m = (2 * (mn % P.tiles_m) + rank) * CTA_ROWS + row;
            const int n0 = (mn / P.tiles_m) * BN_ + half * COLS;
            if (row < CTA_ROWS && m < P.M_total) {
                float *p = P.out + (long long)(t / tiles_mn) * P.split_stride + m * P.m_stride + n0 * P.n_stride;
                const long long step = P.n_stride;
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    const int ncols = P.N_total - (n0 + c * 32);
                    if (ncols >= 32 && step == 1 && !P.accumulate && ((uintptr_t)p & 15) == 0) {
#pragma unroll
                        for (int j = 0; j < 32; j += 4) *(float4 *)(p + j) = make_float4(__fadd_rn(0.f, acc[c][j]), __fadd_rn(0.f, acc[c][j + 1]), __fadd_rn(0.f, acc[c][j + 2]), __fadd_rn(0.f, acc[c][j + 3]));
                    } else if (ncols >= 32 && !P.accumulate) {
                        float *q = p;
#pragma unroll
                        for (int j = 0; j < 32; j++) { *q = __fadd_rn(0.f, acc[c][j]); q += step; }
                    } else if (P.accumulate) {
                        // eight old values at a time: a load cannot be moved above the store before it, and one by one the 64 round
                        // trips of a row are longer than the reduction of a small layer (48 x 720 channels, 10 x 8, one image: 41 us)
#pragma unroll
                        for (int h = 0; h < 32; h += 8) {
                            float prev[8];
#pragma unroll
                            for (int j = 0; j < 8; j++) prev[j] = h + j < ncols ? __ldcg(p + (h + j) * step) : 0.f;
#pragma unroll
                            for (int j = 0; j < 8; j++) if (h + j < ncols) p[(h + j) * step] = __fadd_rn(prev[j], acc[c][h + j]);
                        }
                    } else {
                        float *q = p;
#pragma unroll
                        for (int j = 0; j < 32; j++)
                            if (j < ncols) { *q = __fadd_rn(0.f, acc[c][j]); q += step; }
                    }
                    p += 32 * step;
                }
            }
            __syncwarp();
        }
    }
    // status word: site of the first wait that gave up | warp << 8 | 6 << 16 (this kernel)
    if (failed) { *abort_flag = 1; atomicCAS(P.status, 0, fail_code | (warp << 8) | (6 << 16)); }
    tc_fence_before();
    __syncthreads();
    // both CTAs are done with each other's barriers, shared memory and accumulators
    cluster_arrive(); cluster_wait();
    if (warp == 8) tmem_dealloc_pair(tmem_base, 512);
}

}  // namespace

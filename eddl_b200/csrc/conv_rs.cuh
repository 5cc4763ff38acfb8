// Row-shift convolution: forward and backward-data of Conv2D on pairs of CTAs (tcgen05.mma, cta_group::2).
//
// What bounds a 3xTF32 convolution on this GPU is not the tensor pipe but shared-memory bandwidth (128 bytes per SM and cycle).
// For a 128 x 128 tile, a K-block of 32 costs 12 MMAs of 64 cycles; with one operand tile per filter tap and one CTA per tile
// the same K-block moves 384 cycles' worth of bytes through the conversion of the activations (load, split, two stores), 768 through
// the MMAs' operand reads and 256 through the copy of the weights: 1408 cycles by this count (not all of it in a row: about 1300 measured).
// Here
//   * the activations are converted ONCE per 32-channel group, not once per tap.  Pixels are numbered in a padded space: image
//     rows of pitch Wp (the image width plus the larger of the two side paddings), images of Hp rows, the padding reading as
//     zero.  In that space a filter tap is a constant shift, and shared memory holds a SLAB of the group: one 128-byte row of 32
//     channels per position (K-major, 128-byte swizzle), the tile's 128 positions plus the halo of the shifts.  The operand
//     of a tap is the slab read from `shift` rows further on: the swizzle is a function of address bits, so a matrix descriptor
//     may start at any row (all shifts checked on the hardware), and nine taps share one conversion;
//   * two CTAs of a cluster work on 256 positions x BN filters with M = 256 instructions: each holds its own 128 positions and HALF
//     of the weights, which halves the traffic of the weight copies and a quarter of the operand reads.
// Per K-block and SM: conversion 81 cycles (56 x 56 images), operand reads 576, weights 128 -- 785, just above the 768 of the
// MMAs; measured 833 with fill and drain, the tensor pipe busy 92 % of the time (profiles/conv_pairs_bn_gemm.md).  64 x 256 x 56 x 56,
// 256 filters, 3 x 3 forward, igemm_tc_kernel -> this kernel: single launches behind a flushed L2 1.04 -> 0.81 ms; back to back
// for a second, where the power cap holds the SM clock at 1.53 GHz, 0.93 ms (run_rs has the rule for where it is used).
//
// Positions run across images, so planes of any size and width fill whole tiles (what is lost is the padding: 1 column per row and
// 1 row per image), the halo is read with plain loads and the channel count need not be a multiple of anything.  Strides:
// a forward layer of stride 2 reads one slab per phase (row and column parity) of its input, a backward-data layer of stride 2 is
// one dense problem per parity class of dx, all of them in one launch.
//
//   warps 0-7    converters: two groups of four warps take alternate slabs; a thread owns a position and has the group's 32
//                channels in registers while the slab buffer it will fill is still being read by MMAs.
//   warp  8      (first CTA of the pair) one lane issues the MMAs.
//   warp  9      one lane fetches this CTA's half of each K-block's weights by TMA; the bytes of both CTAs are counted on the
//                first CTA's barrier.
//   warps 10-17  epilogue: two warps per TMEM lane quarter, half of the filters each.
// Every wait is bounded as in igemm_tc_kernel.
#pragma once
#include "tc_ptx.cuh"

namespace {

using namespace eb;

constexpr int RS_THREADS = 18 * 32;
constexpr int RS_MAX_TAPS = 64, RS_MAX_SLABS = 4, RS_MAX_BUF = 4, RS_MAX_BST = 8;
constexpr int RS_BAR_WORDS = 2 * RS_MAX_BUF + 2 * RS_MAX_BST + 4;
constexpr int RS_SMEM_LIMIT = 232448;
constexpr uint32_t RS_SLAB_BEGIN = 1u << 20, RS_SLAB_END = 1u << 21, RS_TILE_BEGIN = 1u << 22, RS_TILE_END = 1u << 23, RS_LAST = 1u << 24;

struct RsSlab { int min_shift, rows, tap0, ntaps, rho, sigma; };          // one per input phase (forward) or class (backward-data)
struct RsClass { int slab0, nslabs, taps, kb_base, dh, dw, y0, x0; };      // an output class: its slabs and where its pixels lie
struct RsParams {
    CUtensorMap mapB;
    const float *src, *bias;
    float *out, *part;
    int *status;
    int images, C, sh, sw, ssr, ssc;          // source tensor and the step between the pixels of one phase
    int Wp, img_pos, M_total;                 // padded space: row pitch, positions per image, positions in all
    int K, dhw, dw_full, dsr, dsc;            // destination tensor
    int tiles_m, tiles_n, splits, ncls, cgs, nmain;
    int accumulate, add_zero;
    int slab_plane, nbuf, bst;                // bytes of one slab plane, slab buffers, weight stages
    RsClass cls[RS_MAX_SLABS];
    RsSlab slab[RS_MAX_SLABS];
    short tap_row[RS_MAX_TAPS];               // rows from the start of the slab to the tap's operand
};

// Walks the slabs of the CTA pair's tile sequence: all roles step through it in the same order.
struct RsWalk {
    int t, kb0, kb1, cg, ph, t0, t1;          // tile; its K-blocks; channel group, slab of the class, taps [t0, t1) of the slab in this tile
    const RsClass *c;
    __device__ __forceinline__ void open(const RsParams &P, int tile) {
        t = tile;
        const int per = P.tiles_m * P.tiles_n * P.splits, cl = P.ncls > 1 ? tile / per : 0, split = tile % P.splits;
        c = &P.cls[cl];
        const int nkb = c->taps * P.cgs;
        kb0 = (int)((long long)split * nkb / P.splits); kb1 = (int)((long long)(split + 1) * nkb / P.splits);
        cg = kb0 / c->taps; ph = -1;
    }
    // next slab with work in the current tile; false = tile done
    __device__ __forceinline__ bool next(const RsParams &P) {
        for (;;) {
            if (++ph == c->nslabs) { ph = 0; cg++; }
            const int base = cg * c->taps;
            if (base >= kb1) return false;
            const RsSlab &s = P.slab[c->slab0 + ph];
            const int first = s.tap0 - P.slab[c->slab0].tap0;               // number of the slab's first tap inside the class
            t0 = max(kb0 - base - first, 0); t1 = min(kb1 - base - first, s.ntaps);
            if (t0 < t1) return true;
        }
    }
    __device__ __forceinline__ int m_tile(const RsParams &P) const { return (t / (P.splits * P.tiles_n)) % P.tiles_m; }
    __device__ __forceinline__ int n_tile(const RsParams &P) const { return (t / P.splits) % P.tiles_n; }
};

template <int BN_, int PREC>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(RS_THREADS, 1) conv_rs_kernel(const __grid_constant__ RsParams P) {
    constexpr bool SPLIT3 = PREC != 1, CROSS_BF16 = PREC == 2;
    constexpr int PLANES = SPLIT3 ? 2 : 1;
    constexpr int B_HALF = BN_ / 2 * 128;                    // one plane of this CTA's half of a K-block's weights
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int slab_bytes = P.slab_plane * PLANES;
    uint8_t *b_base = smem + P.nbuf * slab_bytes;
    uint64_t *bars = (uint64_t *)(b_base + P.bst * PLANES * B_HALF);
    uint32_t *tmem_slot = (uint32_t *)(bars + RS_BAR_WORDS);
    volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
    volatile uint32_t *stage_word = tmem_slot + 2;           // what the K-block in a weight stage is (first CTA), see the MMA issuer
    const uint32_t bar_slab_full = smem_u32(bars), bar_slab_empty = bar_slab_full + 8 * RS_MAX_BUF;
    const uint32_t bar_b_full = bar_slab_empty + 8 * RS_MAX_BUF, bar_b_empty = bar_b_full + 8 * RS_MAX_BST;
    const uint32_t bar_acc_full = bar_b_empty + 8 * RS_MAX_BST, bar_acc_empty = bar_acc_full + 16;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_rank();
    const int pair = (int)(blockIdx.x >> 1), pairs = (int)(gridDim.x >> 1);
    const int total_tiles = P.ncls * P.tiles_m * P.tiles_n * P.splits;
    const int nacc = P.nmain + (SPLIT3 ? 1 : 0), set_cols = nacc * BN_, nsets = 512 / set_cols >= 2 ? 2 : 1;

    if (tid == 0) {
        for (int s = 0; s < P.nbuf; s++) { mbar_init(bar_slab_full + 8 * s, 8); mbar_init(bar_slab_empty + 8 * s, 1); }      // four warps of each CTA
        for (int s = 0; s < P.bst; s++) { mbar_init(bar_b_full + 8 * s, 1); mbar_init(bar_b_empty + 8 * s, 1); }
        for (int s = 0; s < 2; s++) { mbar_init(bar_acc_full + 8 * s, 1); mbar_init(bar_acc_empty + 8 * s, 16); }            // eight warps of each CTA
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8) tmem_alloc_pair(smem_u32(tmem_slot), 512);
    EB_GRID_WAIT();
    tc_fence_before();
    __syncthreads();
    cluster_arrive(); cluster_wait();                        // the other CTA's barriers are initialised before anything arrives on them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    bool failed = false;
    int fail_code = 0;

    if (warp < 8) {
        // ============================ converters ============================
        const int group = warp >> 2, gtid = tid & 127;
        const uint32_t full_of_first = map_to_rank(bar_slab_full, 0);
        RsWalk w;
        int t = pair, sq = -1;                               // sq: number of the slab in the CTA's sequence
        bool open = false;
        // step to the next slab that belongs to this group; false = no more
        auto advance = [&]() -> bool {
            for (;;) {
                if (!open) { if (t >= total_tiles) return false; w.open(P, t); open = true; }
                if (!w.next(P)) { open = false; t += pairs; continue; }
                if (((++sq) & 1) == group) return true;
            }
        };
        float av[BK];
        const int shw = P.sh * P.sw;
        auto load = [&](int row) {
            const RsSlab &s = P.slab[w.c->slab0 + w.ph];
            const int c0 = w.cg * BK, nc = min(P.C - c0, BK);
            const int pos = w.m_tile(P) * 256 + (int)rank * 128 + s.min_shift + row;
            const int img = pos >= 0 ? pos / P.img_pos : -1, rem = pos - img * P.img_pos, y = rem / P.Wp, x = rem - y * P.Wp;
            const int sy = y * P.ssr + s.rho, sx = x * P.ssc + s.sigma;
            const bool ok = pos >= 0 && img < P.images && sy < P.sh && sx < P.sw && row < s.rows;
            const float *q = P.src + ((size_t)(ok ? img : 0) * P.C + c0) * shw + (ok ? sy * P.sw + sx : 0);
            if (nc == BK) {
#pragma unroll
                for (int i = 0; i < BK; i++) av[i] = ok ? __ldg(q + (size_t)i * shw) : 0.f;
            } else {
#pragma unroll
                for (int i = 0; i < BK; i++) av[i] = ok && i < nc ? __ldg(q + (size_t)i * shw) : 0.f;
            }
        };
        auto store = [&](uint8_t *hi_plane, int row) {
            const int nc8 = (P.C - w.cg * BK + 7) & ~7;
            uint8_t *lo_plane = hi_plane + P.slab_plane;         // only when SPLIT3
            if (CROSS_BF16) {
#pragma unroll
                for (int g = 0; g < BK / 8; g++) {
                    float hi[8], lo[8];
#pragma unroll
                    for (int j = 0; j < 8; j++) split_tf32(av[8 * g + j], hi[j], lo[j]);
                    *(float4 *)(hi_plane + swz(row, g * 8)) = make_float4(hi[0], hi[1], hi[2], hi[3]);
                    *(float4 *)(hi_plane + swz(row, g * 8 + 4)) = make_float4(hi[4], hi[5], hi[6], hi[7]);
                    *(uint4 *)(lo_plane + swz_chunk(row, g)) = make_uint4(pack_bf16(lo[0], lo[1]), pack_bf16(lo[2], lo[3]), pack_bf16(lo[4], lo[5]), pack_bf16(lo[6], lo[7]));
                    *(uint4 *)(lo_plane + swz_chunk(row, 4 + g)) = make_uint4(pack_bf16(hi[0], hi[1]), pack_bf16(hi[2], hi[3]), pack_bf16(hi[4], hi[5]), pack_bf16(hi[6], hi[7]));
                }
            } else {
#pragma unroll
                for (int g = 0; g < BK / 4; g++) {
                    if (4 * g >= nc8) break;             // channels past the last one: only what its k-step reads is written (zeros)
                    const uint32_t off = swz(row, g * 4);
                    if (SPLIT3) {
                        float4 hi, lo;
                        split_tf32(av[4 * g], hi.x, lo.x); split_tf32(av[4 * g + 1], hi.y, lo.y); split_tf32(av[4 * g + 2], hi.z, lo.z); split_tf32(av[4 * g + 3], hi.w, lo.w);
                        *(float4 *)(hi_plane + off) = hi; *(float4 *)(lo_plane + off) = lo;
                    } else *(float4 *)(hi_plane + off) = make_float4(av[4 * g], av[4 * g + 1], av[4 * g + 2], av[4 * g + 3]);
                }
            }
        };
        bool more = advance();
        if (more) load(gtid);
        while (more) {
            const int buf = sq % P.nbuf;
            if (!mbar_wait_warp(bar_slab_empty + 8 * buf, ((sq / P.nbuf) & 1) ^ 1, abort_flag)) { failed = true, fail_code = 1; break; }
            uint8_t *plane = smem + buf * slab_bytes;
            const int rows = P.slab[w.c->slab0 + w.ph].rows;
            store(plane, gtid);                              // a slab has at least 128 rows
            for (int row = gtid + 128; row - gtid < rows; row += 128) {
                load(row);
                if (row * 128 < P.slab_plane) store(plane, row);
            }
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(full_of_first + 8 * buf);
            more = advance();
            if (more) load(gtid);
        }
    } else if (warp == 8) {
        // ============================ MMA issuer (one lane of the first CTA) ============================
        // As in igemm_tc_kernel nothing in the loop waits for a result between MMAs.  What a K-block is -- the row of the slab where
        // its tap's operand starts, how many k-steps, whether a slab or a tile begins or ends -- is worked out by the weight
        // warp, which leaves one word per weight stage beside the stage; this thread reads the word of the NEXT stage, and looks
        // at its barriers, in the middle of a K-block.
        if (rank == 0 && elect_one()) {
            constexpr uint32_t idesc = make_idesc_pair(BN_);
            constexpr uint32_t DESC_HI = 64u | (1u << 14) | (2u << 29);            // upper word of make_desc()
            auto desc = [&](uint32_t lo) { return ((uint64_t)DESC_HI << 32) | lo; };
            const uint32_t a0_lo = ((smem_u32(smem) >> 4) & 0x3FFFu) | (1u << 16), b0_lo = ((smem_u32(b_base) >> 4) & 0x3FFFu) | (1u << 16);
            const uint32_t slab_step = (uint32_t)slab_bytes >> 4, plane_step = (uint32_t)P.slab_plane >> 4;
            constexpr uint32_t STAGE_STEP = (uint32_t)(PLANES * B_HALF) >> 4, B_STEP = (uint32_t)B_HALF >> 4;
            const int nmain = P.nmain;
            const uint32_t rot_step = nmain > 1 ? (uint32_t)BN_ : 0u;
            const uint32_t nbuf = (uint32_t)P.nbuf, bst = (uint32_t)P.bst;
            uint32_t buf = 0, buf_phase = 0, s = 0, phase = 0, set_phase = 1, ready = 0, word = 0, a_slab = 0;
            uint32_t d0 = 0, d1 = 0, d2 = 0, d_small = 0;
            int set = 0, steps = 0;                          // k-steps issued in this tile
            if (pair < total_tiles) {
                if (!mbar_wait(bar_b_full, 0u, abort_flag)) failed = true, fail_code = 4;
                else { ready = 1; word = stage_word[0]; }
            }
            while (ready && !failed) {
                const uint32_t w = word;
                if (w & RS_TILE_BEGIN) {
                    if (!mbar_wait(bar_acc_empty + 8 * set, set_phase, abort_flag)) { failed = true, fail_code = 2; break; }
                    d0 = tmem_base + (uint32_t)(set * set_cols); d1 = d0 + rot_step; d2 = d1 + rot_step; d_small = d0 + (uint32_t)(nmain * BN_);
                    steps = 0;
                }
                if (w & RS_SLAB_BEGIN) {
                    if (!mbar_wait(bar_slab_full + 8 * buf, buf_phase, abort_flag)) { failed = true, fail_code = 3; break; }
                    a_slab = a0_lo + buf * slab_step;
                }
                tc_fence_after();
                const uint32_t a_hi = a_slab + 8u * (w & 0xffffu), a_lo = a_hi + plane_step, b_hi = b0_lo + s * STAGE_STEP, b_lo = b_hi + B_STEP;
                const uint32_t next_s = s + 1 == bst ? 0u : s + 1, next_phase = phase ^ (s + 1 == bst ? 1u : 0u);
                // the next stage's word may be read once its barrier has completed
                auto look = [&]() { if ((ready = mbar_test(bar_b_full + 8 * next_s, next_phase)) != 0) word = stage_word[next_s]; };
                const uint32_t ksteps = (w >> 16) & 7u;
                if (ksteps == BK / 8) {
#pragma unroll
                    for (int ks = 0; ks < BK / 8; ks++) {
                        const uint32_t o = 2u * ks;
                        if (SPLIT3 && !CROSS_BF16) {
                            umma_tf32_pair(d_small, desc(a_lo + o), desc(b_hi + o), idesc, ks || steps ? 1u : 0u);
                            umma_tf32_pair(d_small, desc(a_hi + o), desc(b_lo + o), idesc, 1u);
                        }
                        if (CROSS_BF16) umma_bf16_pair(d_small, desc(a_lo + o), desc(b_lo + o), make_idesc_bf16_pair(BN_), ks || steps ? 1u : 0u);
                        umma_tf32_pair(ks == 1 ? d1 : ks == 2 ? d2 : d0, desc(a_hi + o), desc(b_hi + o), idesc, steps + ks >= nmain ? 1u : 0u);
                        if (ks == 1) look();
                    }
                    const uint32_t first = d0;
                    d0 = d1; d1 = d2; d2 = first;
                } else {
                    // the last, partly filled channel group
#pragma unroll 1
                    for (uint32_t ks = 0; ks < (CROSS_BF16 ? BK / 8 : ksteps); ks++) {
                        const uint32_t o = 2u * ks;
                        // cross terms in bf16: the 64 columns [lo | hi] x [hi | lo], 16 per instruction, whatever the channel count
                        if (CROSS_BF16) umma_bf16_pair(d_small, desc(a_lo + o), desc(b_lo + o), make_idesc_bf16_pair(BN_), ks || steps ? 1u : 0u);
                        if (ks >= ksteps) continue;
                        if (SPLIT3 && !CROSS_BF16) {
                            umma_tf32_pair(d_small, desc(a_lo + o), desc(b_hi + o), idesc, ks || steps ? 1u : 0u);
                            umma_tf32_pair(d_small, desc(a_hi + o), desc(b_lo + o), idesc, 1u);
                        }
                        umma_tf32_pair(d0, desc(a_hi + o), desc(b_hi + o), idesc, steps + (int)ks >= nmain ? 1u : 0u);
                        const uint32_t first = d0;
                        d0 = d1; d1 = d2; d2 = first;
                    }
                    look();
                }
                steps += (int)ksteps;
                umma_commit_pair(bar_b_empty + 8 * s);
                if (w & RS_SLAB_END) {
                    umma_commit_pair(bar_slab_empty + 8 * buf);
                    if (++buf == nbuf) { buf = 0; buf_phase ^= 1u; }
                }
                if (w & RS_TILE_END) {
                    umma_commit_pair(bar_acc_full + 8 * set);
                    if (++set == nsets) { set = 0; set_phase ^= 1u; }
                    if (w & RS_LAST) break;
                }
                s = next_s; phase = next_phase;
                if (!ready) {
                    if (!mbar_wait(bar_b_full + 8 * s, phase, abort_flag)) { failed = true, fail_code = 4; break; }
                    ready = 1; word = stage_word[s];
                }
            }
        }
        __syncwarp();
    } else if (warp == 9) {
        // ============================ weights (one lane of each CTA) ============================
        if (lane == 0) {
            const uint32_t full_of_first = map_to_rank(bar_b_full, 0);
            int s = 0, uses = 0; uint32_t phase = 1;
            RsWalk w;
            for (int t = pair; t < total_tiles && !failed; t += pairs) {
                w.open(P, t);
                const int n_tile = w.n_tile(P);
                int kb = w.kb0;
                while (!failed && w.next(P)) {
                    const int tap0 = P.slab[w.c->slab0 + w.ph].tap0, ksteps = min((P.C - w.cg * BK + 7) >> 3, BK / 8);
                    for (int tap = w.t0; tap < w.t1; tap++, kb++) {
                        if (!mbar_wait(bar_b_empty + 8 * s, phase, abort_flag)) { failed = true, fail_code = 5; break; }
                        if (rank == 0) {
                            stage_word[s] = (uint32_t)P.tap_row[tap0 + tap] | (uint32_t)ksteps << 16 | (tap == w.t0 ? RS_SLAB_BEGIN : 0u) | (tap + 1 == w.t1 ? RS_SLAB_END : 0u) |
                                            (kb == w.kb0 ? RS_TILE_BEGIN : 0u) | (kb + 1 == w.kb1 ? RS_TILE_END | (t + pairs >= total_tiles ? RS_LAST : 0u) : 0u);
                            mbar_expect_tx(bar_b_full + 8 * s, 2u * PLANES * B_HALF);          // the bytes of both CTAs
                        }
                        const int row = ((w.c->kb_base + kb) * P.tiles_n + n_tile) * (PLANES * BN_) + (int)rank * (BN_ / 2);
                        const uint32_t dst = smem_u32(b_base) + (uint32_t)(s * PLANES * B_HALF);
                        tma_load_2d_pair(dst, &P.mapB, 0, row, full_of_first + 8 * s);
                        if (SPLIT3) tma_load_2d_pair(dst + B_HALF, &P.mapB, 0, row + BN_, full_of_first + 8 * s);
                        uses++;
                        if (++s == P.bst) { s = 0; phase ^= 1u; }
                    }
                }
            }
            // the last arrivals on this CTA's stage barriers come from the other CTA: stay until they are in
            for (int i = 0; i < P.bst && i < uses && !failed; i++) {
                if (--s < 0) { s = P.bst - 1; phase ^= 1u; }
                if (!mbar_wait(bar_b_empty + 8 * s, phase ^ 1u, abort_flag)) { failed = true, fail_code = 6; }
            }
        }
        __syncwarp();
    } else {
        // ============================ epilogue (warps 10-17) ============================
        const int quarter = warp & 3, half = (warp - 10) >> 2;
        constexpr int COLS = BN_ >= 64 ? BN_ / 2 : 32, NC = COLS / 32;          // BN = 32: the second half has nothing to drain
        const uint32_t empty_of_first = map_to_rank(bar_acc_empty, 0);
        int set = 0; uint32_t set_phase = 0;
        RsWalk w;
        for (int t = pair; t < total_tiles; t += pairs) {
            w.open(P, t);
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
            const int n_tile = w.n_tile(P), m_tile = w.m_tile(P);
            if (P.splits > 1) {
                // leave the partial sums as [filter][128 positions] per tile, CTA and split: rs_combine_kernel adds them
                const size_t tile = (size_t)(t / P.splits) * 2 + rank;
                float *mine = P.part + (tile * P.splits + t % P.splits) * (BN_ * 128) + (half * COLS) * 128 + quarter * 32 + lane;
#pragma unroll
                for (int c = 0; c < NC; c++)
#pragma unroll
                    for (int j = 0; j < 32; j++) __stcg(mine + (c * 32 + j) * 128, acc[c][j]);
                continue;
            }
            const int pos = m_tile * 256 + (int)rank * 128 + quarter * 32 + lane;
            const int img = pos / P.img_pos, rem = pos - img * P.img_pos, y = rem / P.Wp, x = rem - y * P.Wp;
            if (pos < P.M_total && y < w.c->dh && x < w.c->dw) {
                const int col0 = n_tile * BN_ + half * COLS;
                float *p = P.out + ((size_t)img * P.K + col0) * P.dhw + (size_t)(w.c->y0 + y * P.dsr) * P.dw_full + (w.c->x0 + x * P.dsc);
                const size_t step = P.dhw;
    #pragma unroll
                for (int c = 0; c < NC; c++) {
                    const int ncols = P.K - (col0 + c * 32);
                    if (ncols >= 32) {
                        if (P.accumulate) {
                            const float *q = p;
#pragma unroll
                            for (int h = 0; h < 32; h += 8) {
                                float prev[8];
#pragma unroll
                                for (int j = 0; j < 8; j++) { prev[j] = __ldcg(q); q += step; }
#pragma unroll
                                for (int j = 0; j < 8; j++) { *p = __fadd_rn(prev[j], acc[c][h + j]); p += step; }
                            }
                        } else if (P.bias) {
    #pragma unroll
                            for (int j = 0; j < 32; j++) { *p = __fadd_rn(acc[c][j], __ldg(P.bias + col0 + c * 32 + j)); p += step; }
                        } else if (P.add_zero) {
    #pragma unroll
                            for (int j = 0; j < 32; j++) { *p = __fadd_rn(0.f, acc[c][j]); p += step; }
                        } else {
    #pragma unroll
                            for (int j = 0; j < 32; j++) { *p = acc[c][j]; p += step; }
                        }
                    } else {
    #pragma unroll
                        for (int j = 0; j < 32; j++)
                            if (j < ncols) {
                                float v = acc[c][j];
                                if (P.accumulate) v = __fadd_rn(__ldcg(p), v);
                                else if (P.bias) v = __fadd_rn(v, __ldg(P.bias + col0 + c * 32 + j));
                                else if (P.add_zero) v = __fadd_rn(0.f, v);
                                *p = v; p += step;
                            }
                    }
                }
            }
            __syncwarp();
        }
    }
    // status word: site of the first wait that gave up | warp << 8 | 5 << 16 (this kernel)
    if (failed) { *abort_flag = 1; atomicCAS(P.status, 0, fail_code | (warp << 8) | (5 << 16)); }
    tc_fence_before();
    __syncthreads();
    // both CTAs are done with each other's barriers, shared memory and accumulators
    cluster_arrive(); cluster_wait();
    if (warp == 8) tmem_dealloc_pair(tmem_base, 512);
}

// Sum of the splits' partial sums, in order, and the store of the result: out[...] = (accumulate ? out : 0) + sum (+ bias).  One thread
// per position and filter, 128 consecutive positions per group of threads, so reads and writes are coalesced; as a launch of
// its own the partial sums of a tile are read by the whole GPU, not by the one SM that would finish the tile.
template <int BN_>
__global__ void __launch_bounds__(256) rs_combine_kernel(const __grid_constant__ RsParams P) {
    EB_GRID_WAIT();
    const int row = threadIdx.x & 127, sub = threadIdx.x >> 7;
    const int half_tile = blockIdx.x, tile = half_tile >> 1, rank = half_tile & 1;            // tile: (class, position tile, filter tile)
    const int n_tile = tile % P.tiles_n, m_tile = (tile / P.tiles_n) % P.tiles_m, cl = tile / (P.tiles_n * P.tiles_m);
    const RsClass &c = P.cls[cl];
    const int pos = m_tile * 256 + rank * 128 + row;
    const int img = pos / P.img_pos, rem = pos - img * P.img_pos, y = rem / P.Wp, x = rem - y * P.Wp;
    if (pos >= P.M_total || y >= c.dh || x >= c.dw) return;
    const float *part = P.part + (size_t)half_tile * P.splits * (BN_ * 128) + row;
    float *out = P.out + (size_t)img * P.K * P.dhw + (size_t)(c.y0 + y * P.dsr) * P.dw_full + (c.x0 + x * P.dsc);
    for (int col = blockIdx.y * 8 + sub; col < blockIdx.y * 8 + 8; col += 2) {
        const int f = n_tile * BN_ + col;
        if (f >= P.K) return;
        float s = 0.f;
#pragma unroll 8
        for (int z = 0; z < P.splits; z++) s += __ldcg(part + (size_t)z * (BN_ * 128) + col * 128);
        float *q = out + (size_t)f * P.dhw;
        if (P.accumulate) s = __fadd_rn(*q, s);
        else if (P.bias) s = __fadd_rn(s, __ldg(P.bias + f));
        *q = s;
    }
}

}  // namespace

// conv_tc_kernel<MODE, KIND>: the general tcgen05 implicit-GEMM convolution kernel (forward, input gradient by parity
// class, kernel gradient; TF32 and 3xTF32).  Included by conv_tc.cu only.
#pragma once

namespace dcg {
namespace {

// ---- 3xTF32: blocks of stages ---------------------------------------------------------------------
// The short chains used to come from eight K partitions per tile, each a CTA with its set-up, its partial tile through L2
// and its epilogue; now a CTA sums blocks of stages in registers and the partitions follow the SM count as for plain
// TF32.  Measured, 128 -> 256 channels at batch 64: forward 91 -> 49 us, input gradient 124 -> 61, kernel gradient
// 80 -> 57; relative error against float64 4e-7 at every layer (3.6e-7 to 4.7e-6 before).
constexpr int kX3Block = 4;   // K stages per block: sixteen truncating steps in a row

// Kinds of launch.
//   kShared   the plain one; two CTAs per SM where the grid is large enough
//   kX3       3xTF32, up to 128 columns
//   kX3Wide   3xTF32, up to 192 columns (the kernel gradient of an RGB layer)
//   kAlone    one CTA per SM and no K partitions: more threads for the epilogue (64 -> 128 forward of 64 images 16.6 -> 15.5
//             us; with partitions the cluster barrier of the larger CTA costs more, +0.6 to 1 us)
//   kDual     one CTA per SM and at most 64 columns: the MMAs of a stage are too short to cover the hand-over to the next, so
//             two warps issue them in turn, each into an accumulator of its own, and two warps load (64 -> 128 kernel
//             gradient of 64 images 22.9 -> 20.4 us; from 128 columns on there was nothing to gain)
enum Kind { kShared, kX3, kAlone, kDual, kX3Wide, kKinds };
__host__ __device__ constexpr bool is_x3(int kind) { return kind == kX3 || kind == kX3Wide; }
// Groups of four epilogue warps, one warp per TMEM lane quadrant each.  3xTF32: taking a stage apart (2500 clocks, most of them
// waits for shared memory, which the MMAs' operands keep busy) and taking over the sums (1300 every fourth stage) pace the
// loop, so there are as many groups as registers allow: with four, a warp sums one 32-column slab of the tile, with three,
// two.  (Against three throughout: step of 64 images 3095 -> 3058 us, 64 -> 3 input gradient of 64 images 41.3 -> 38.3.)
template <int KIND> constexpr int kGroups = KIND == kX3Wide ? 3 : KIND == kX3 || KIND == kAlone ? 4 : 2;
inline int epilogue_groups(int kind)
{
    static const int groups[kKinds] = {kGroups<kShared>, kGroups<kX3>, kGroups<kAlone>, kGroups<kDual>, kGroups<kX3Wide>};
    return groups[kind];
}
template <int KIND> constexpr int kX3Slabs = KIND == kX3Wide ? 2 : 1;   // slabs per epilogue warp, every kGroups-th one
template <int KIND> constexpr int kX3Width = 32 * kGroups<KIND> * kX3Slabs<KIND>;
constexpr int kX3MaxWidth = kX3Width<kX3Wide>;
// 3xTF32: accumulators of the large terms.
__host__ __device__ constexpr int x3_accumulators(int bn) { return bn <= 128 ? 2 : 1; }
// TMEM columns of a CTA: at most 512, or 256 where two share an SM.
__host__ __device__ constexpr int tmem_columns(int kind, int bn, int x3_slots)
{
    return is_x3(kind) ? (x3_accumulators(bn) + 1) * bn + 64 * x3_slots : kind == kDual ? 2 * bn : bn;
}

// Adds the accumulator's slabs of this warp to `sum`.
template <int KIND>
__device__ __forceinline__ void x3_take_over(float (&sum)[kX3Slabs<KIND>][32], uint32_t tmem_quad, int group, int bn)
{
#pragma unroll
    for (int sl = 0; sl < kX3Slabs<KIND>; ++sl) {
        const int c0 = group * 32 + sl * 32 * kGroups<KIND>;
        if (c0 < bn) {
            uint32_t r[32];
            const bool full = bn - c0 >= 32;
            if (full) tmem_ld_32x32b_x32(tmem_quad + (uint32_t)c0, r);
            else tmem_ld_32x32b_x16(tmem_quad + (uint32_t)c0, r);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int q = 0; q < 32; ++q)
                if (q < 16 || full) sum[sl][q] = __fadd_rn(sum[sl][q], __uint_as_float(r[q]));
        }
    }
}

// ---- the kernel ---------------------------------------------------------------------------------
// TAPS (kernel gradient only): kernel taps whose input channels share the 128 rows of an M tile.  A template argument, for a
// run-time choice takes the coordinates of the loads out of uniform registers (128 -> 256 gradient of 64 images 18.7 -> 21.6 us).
// 0: one tap, with the MN-major operands of ragged channel counts loaded in pieces of 32 channels.
template <int MODE, int KIND, int TAPS = 1>
__global__ void __launch_bounds__(64 + 128 * kGroups<KIND>, KIND == kShared ? 2 : 1)
conv_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
               const __grid_constant__ Params p)
{
    constexpr bool X3 = is_x3(KIND), PIECES = TAPS == 0;
    constexpr int MT = PIECES ? 1 : TAPS;
    // Warps that take the stages in turn, as producers and as MMA issuers.  With two of them the ring has an even number of
    // stages: a stage is then always the same warp's, which makes the parity of its barriers unambiguous.
    constexpr int W = KIND == kDual ? 2 : 1;
    constexpr int G = kGroups<KIND>, EPI = 128 * G;   // epilogue threads
    extern __shared__ uint8_t smem_raw[];
    if (threadIdx.x == 64) TC_TRACE(3072);
    TC_CTA_TRACE(0);
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int b_stage_bytes = p.bn * BK * 4;
    const long long wait_limit = p.wait_cycles;
    const uint32_t a_base = smem_base;
    const uint32_t b_base = a_base + (uint32_t)p.stages * A_STAGE_BYTES;
    // 3xTF32: residual tiles of B (operand minus its TF32 part) follow the operand tiles; A and its residual go to TMEM
    const uint32_t bs_base = b_base + (uint32_t)p.stages * b_stage_bytes;
    const uint32_t bar_base = X3 ? bs_base + (uint32_t)p.x3_bslots * b_stage_bytes : bs_base;
    // barriers: full[stages], empty[stages], tmem_full; then the TMEM base address word
    const uint32_t full_bar = bar_base;
    const uint32_t empty_bar = bar_base + 8u * p.stages;
    const uint32_t resid_bar = bar_base + 16u * p.stages;     // 3xTF32: residual tiles of the stage are written
    const uint32_t tmem_full_bar = bar_base + 24u * p.stages;
    const uint32_t tmem_slot = tmem_full_bar + 8u;
    const uint32_t promo_full_bar = tmem_full_bar + 16u;      // 3xTF32, [2]: a block of kX3Block stages is summed ...
    const uint32_t promo_empty_bar = tmem_full_bar + 32u;     // ... [2] and taken over into registers
    uint32_t* tmem_slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

    // ---- one-time setup -------------------------------------------------------------------------------
    // With one CTA per SM nothing hides it: a CTA starts when its predecessor's has left.  So its steps are kept short - a lane
    // per stage for the barriers, no division by run-time values - and everything that does not touch memory comes before the
    // wait for the launch before (from a CTA's start to its first load it was 1.6 to 2.2 us: 64 -> 128 forward of 8 images 8.2 -> 7.3,
    // of 64 images 16.2 -> 15.7 us).
    if (warp == 0) {
        if (lane < p.stages) {
            mbar_init(full_bar + 8u * lane, 1);
            mbar_init(empty_bar + 8u * lane, 1);
            if (X3) mbar_init(resid_bar + 8u * lane, 128);
        }
        if (X3 && lane < 2) {
            mbar_init(promo_full_bar + 8u * lane, 1);
            mbar_init(promo_empty_bar + 8u * lane, EPI);
        }
        if (lane == 0) {
            mbar_init(tmem_full_bar, W);
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        __syncwarp();
    }
    // 3xTF32 keeps the two small cross terms in an accumulator of their own: the tensor core rounds its
    // accumulator toward zero at every step, an error that grows with the number of steps and with the
    // accumulator's size, so the small terms round among themselves.  The accumulator of the large terms is added (round to
    // nearest) to registers of the epilogue warps after every kX3Block stages; where TMEM has room there are two of
    // it, and the tensor core goes on in the other one.  The A operand is read from TMEM (32 columns of values, 32 of
    // residuals per slot): three MMAs per K step take 12 KB from shared memory instead of 24, which is what would pace
    // the loop.  Columns: x3_mains accumulators, the small terms, x3_slots A slots.
    const int x3_mains = X3 ? x3_accumulators(p.bn) : 1;
    const int x3_a0 = (x3_mains + 1) * p.bn;
    const int x3_slot_mask = p.x3_slots - 1, x3_bslot_mask = p.x3_bslots - 1;   // powers of two
    int tmem_cols = 32;
    while (tmem_cols < tmem_columns(KIND, p.bn, p.x3_slots)) tmem_cols <<= 1;
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }

    // ---- decode this CTA's work item -------------------------------------------------------------
    // blockIdx.x = ((group * m_count + m) * n_tiles + n) * splits + split, where group is the parity
    // class (DX), the kernel tap (DK) or absent (FWD), and m a pixel tile (FWD/DX) or channel tile (DK).
    int rem, split, n_tile, m_tile, group;
    p.by_splits.divmod((int)blockIdx.x, rem, split);
    p.by_n_tiles.divmod(rem, rem, n_tile);
    p.by_m_count.divmod(rem, group, m_tile);

    // pixel-tile origin (FWD/DX)
    int j0 = 0, i0 = 0, n0 = 0;
    if (MODE != MODE_DK) {
        p.by_tiles_w.divmod(m_tile, n0, j0);
        p.by_tiles_h.divmod(n0, n0, i0);
        j0 *= p.TW; i0 *= p.TH; n0 *= p.TN;
    }
    // DX: parity class and its taps; DK: the kernel tap
    int ph = 0, pw = 0, rh = 0, rw = 0, eh = 0, ew = 0, taps_h = 1, taps_w = 1, tap_di = 0, tap_dj = 0;
    if (MODE == MODE_DX) {
        // classes in the order of their first taps, so those with the most taps (9, 6, 6, 4 of 5 x 5 / stride 2) start first and
        // a short one is what fills the last wave
        p.by_sw.divmod(group, rh, rw);
        ph = rh - p.pt_mod; if (ph < 0) ph += p.sh;
        pw = rw - p.pl_mod; if (pw < 0) pw += p.sw;
        eh = p.by_sh.div(ph + p.pt); ew = p.by_sw.div(pw + p.pl);
        taps_h = rh < p.KH ? p.by_sh.div(p.KH - rh + p.sh - 1) : 0;
        taps_w = rw < p.KW ? p.by_sw.div(p.KW - rw + p.sw - 1) : 0;
    } else if (MODE == MODE_DK && !p.narrow) {   // (narrow: columns are 32 window slots per kernel row, all taps in one tile or two)
        p.by_kw.divmod(group * MT, tap_di, tap_dj);   // (the first one)
    }
    // K-stage range of this split: floor(stages * split / splits) on
    int total_stages;
    if (MODE == MODE_FWD) total_stages = p.narrow ? p.KH : p.KH * p.KW * p.kchunks;
    else if (MODE == MODE_DX) total_stages = taps_h * taps_w * p.kchunks;
    else total_stages = p.tiles_w * p.tiles_h * p.tiles_n;
    int each, over;
    p.by_splits.divmod(total_stages, each, over);
    const int q0 = each * split + p.by_splits.div(over * split);
    const int nq = each * (split + 1) + p.by_splits.div(over * (split + 1)) - q0;

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_d = *tmem_slot_ptr;
    // Programmatic dependent launch: everything up to pdl_enter() (barriers, TMEM, descriptor prefetch, the roles' own
    // preparations) may run while the previous kernel of the stream is still draining; the producer and the epilogue
    // warps call it before they touch memory.  The MMA warps only read what the producer has loaded.
    // The next kernel's CTAs may in turn be set up as soon as every CTA of this grid has got there.
    if (threadIdx.x == 64) TC_TRACE(3073);
    TC_CTA_TRACE(1);
#ifdef DCG_TC_TRACING
    if ((p.debug & 8) && threadIdx.x == 64 && blockIdx.x < 1024) {
        unsigned smid;
        asm volatile("mov.u32 %0, %smid;" : "=r"(smid));
        g_tc_cta_trace[blockIdx.x][6] = smid;
    }
#endif

    // ---- epilogue geometry (uniform over the CTA) ---------------------------------------------------
    const int ch0 = n_tile * p.bn;    // channel index of accumulator column 0 (bias axis) unless DK
    int ncols_valid;                  // valid columns in this N tile
    long long col_stride = 1;         // element stride between accumulator columns in the output
    if (MODE == MODE_FWD) ncols_valid = min(p.bn, (p.o_store ? p.o_store : p.O) - ch0);
    else if (MODE == MODE_DX) ncols_valid = min(p.bn, p.C - ch0);
    else if (p.narrow) { ncols_valid = min(p.bn, 32 * p.KH - ch0); col_stride = p.O; }
    else if (!p.swap) ncols_valid = min(p.bn, p.O - ch0);
    else { ncols_valid = min(p.bn, p.C - ch0); col_stride = p.O; }
    // Row-contiguous outputs whose channel count allows 16-byte stores take the vector path.
    const int ch_total = (MODE == MODE_DX) ? p.C : p.O;
    const bool vec = col_stride == 1 && (ch_total & 3) == 0 && (ncols_valid & 3) == 0;
    float* red = reinterpret_cast<float*>(smem_raw + (a_base - smem_u32(smem_raw)));
    long long* s_rowoff = reinterpret_cast<long long*>(red + kRedFloats(p.bn));

    constexpr int SLABS = kX3Slabs<KIND>;
    float x3_sum[SLABS][32];   // 3xTF32: the blocks of stages taken over so far
    if constexpr (X3) {
#pragma unroll
        for (int sl = 0; sl < SLABS; ++sl)
#pragma unroll
            for (int q = 0; q < 32; ++q) x3_sum[sl][q] = 0.f;
    }

    const int walker = warp >> 1;   // kDual: warps 0 and 1 take the even stages; 2 and 3, until their epilogue, the odd ones
    if (warp == 0 || (W == 2 && warp == 2)) {
        // ===== TMA producer =====
        // One thread issues every load.  All position bookkeeping is incremental: an integer division
        // costs this lone thread ~100 cycles, and the loop has to turn around in well under the 256
        // cycles the tensor core needs per stage.
        {
            // MN-major operands of ragged channel counts come in pieces of 32 channels: only those that exist are loaded, what the
            // others leave in their rows and columns is never stored
            const int a_pieces = PIECES && MODE == MODE_DK ? min(BM / 32, (p.a_ch - m_tile * BM + 31) >> 5) : 0;
            const int b_pieces = PIECES ? min(p.bn >> 5, (p.b_ch - n_tile * p.bn + 31) >> 5) : 0;
            const uint32_t tx_bytes = (uint32_t)((MODE != MODE_DK ? p.TW * p.TH * p.TN * BK * 4 : PIECES ? a_pieces * kPieceBytes : A_STAGE_BYTES) +
                                                 (PIECES && !p.narrow ? b_pieces * kPieceBytes : b_stage_bytes));
            int s = walker;
            uint32_t phase = 0;
            // counters of stage q0: FWD (chunk, tap, di, dj); DX (chunk, -, th, tw); DK (-, tile_n, tile_h, tile_w)
            int chunk = 0, tap = 0, di = 0, dj = 0;
            if (MODE == MODE_FWD && !p.narrow) {
                p.by_kchunks.divmod(q0, tap, chunk);
                p.by_kw.divmod(tap, di, dj);
            } else if (MODE == MODE_DX) {
                p.by_kchunks.divmod(q0, di, chunk);
                dj = di;
                for (di = 0; dj >= taps_w && taps_w > 0; ++di) dj -= taps_w;
            } else if (MODE == MODE_DK) {
                p.by_tiles_w.divmod(q0, tap, dj);
                p.by_tiles_h.divmod(tap, tap, di);
            }
            const int wrap_dj = (MODE == MODE_FWD) ? p.KW : taps_w;
            auto advance = [&] {
                if (MODE == MODE_DK) {
                    if (++dj == p.tiles_w) { dj = 0; if (++di == p.tiles_h) { di = 0; ++tap; } }
                } else if (++chunk == p.kchunks) {
                    chunk = 0; ++tap;
                    if (++dj == wrap_dj) { dj = 0; ++di; }
                }
            };
            // DK: where the further taps of an M tile lie, seen from its first one (beyond the last tap: that one again)
            int oh1 = 0, ow1 = 0, oh2 = 0, ow2 = 0, oh3 = 0, ow3 = 0;
            if (MT > 1) {
                const int last = p.KH * p.KW - 1, t1 = min(group * MT + 1, last), t2 = min(group * MT + 2, last), t3 = min(group * MT + 3, last);
                p.by_kw.divmod(t1, oh1, ow1); oh1 -= tap_di; ow1 -= tap_dj;
                p.by_kw.divmod(t2, oh2, ow2); oh2 -= tap_di; ow2 -= tap_dj;
                p.by_kw.divmod(t3, oh3, ow3); oh3 -= tap_di; ow3 -= tap_dj;
            }
            if (walker == 1) advance();
            pdl_enter();
            for (int it = walker; it < nq; it += W) {
                if (!mbar_wait_warp(empty_bar + 8u * s, phase ^ 1u, 0, it, wait_limit)) break;
                const uint32_t fb = full_bar + 8u * s;
                if (it != p.skip_stage && elect_one()) {
                TC_TRACE(it);
                if (TC_DEBUG_BIT(2)) {   // timing experiment: no loads, the stage is declared full at once
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(fb) : "memory");
                } else {
                    mbar_expect_tx(fb, tx_bytes);
                    const uint32_t a_dst = a_base + (uint32_t)s * A_STAGE_BYTES;
                    const uint32_t b_dst = b_base + (uint32_t)s * b_stage_bytes;
                    if (MODE == MODE_FWD && p.narrow) {
                        // stage = kernel row: 128 output pixels x the 32-float window (8 pixels x 4
                        // channels) that starts at padded column s*j of padded row s*i + row
                        const int q = q0 + it;
                        tma_load_5d(a_dst, &map_a, fb, 0, j0, i0, n0, q);
                        tma_load_4d(b_dst, &map_b, fb, 0, 0, q, n_tile * (p.bn / 32));
                    } else if (MODE == MODE_FWD) {
                        if (it < 128) TC_TRACE(256 + it);
                        tma_load_4d(a_dst, &map_a, fb, chunk * BK, p.sw * j0 + dj - p.pl, p.sh * i0 + di - p.pt, n0);
                        if (it < 128) TC_TRACE(512 + it);
                        if constexpr (PIECES) {
                            for (int i = 0; i < b_pieces; ++i)
                                tma_load_4d(b_dst + i * kPieceBytes, &map_b, fb, n_tile * p.bn + 32 * i, chunk * BK, tap, 0);
                        } else {
                            tma_load_4d(b_dst, &map_b, fb, 0, chunk * BK, tap, n_tile * (p.bn / 32));
                        }
                        if (it < 128) TC_TRACE(768 + it);
                    } else if (MODE == MODE_DX) {
                        // (di, dj) count the taps of this parity class: kernel tap (rh + sh*di, rw + sw*dj)
                        tma_load_4d(a_dst, &map_a, fb, chunk * BK, j0 + ew - dj, i0 + eh - di, n0);
                        tma_load_4d(b_dst, &map_b, fb, chunk * BK, n_tile * p.bn, rw + p.sw * dj, rh + p.sh * di);
                    } else {
                        // (tap, di, dj) count the 32-pixel tiles along (n, h, w)
                        const int pj = dj * p.TW, pi = di * p.TH, pn = tap * p.TN;
                        const int xw = p.sw * pj + tap_dj - p.pl, xh = p.sh * pi + tap_di - p.pt;
                        if (p.narrow) {  // A: dy (rows o), B: the 32-float windows of 32 output pixels, one per kernel row
                            if constexpr (PIECES) {
                                for (int i = 0; i < a_pieces; ++i)
                                    tma_load_4d(a_dst + i * kPieceBytes, &map_a, fb, m_tile * BM + 32 * i, pj, pi, pn);
                            } else {
                                tma_load_5d(a_dst, &map_a, fb, 0, pj, pi, pn, m_tile * (BM / 32));
                            }
                            tma_load_5d(b_dst, &map_b, fb, 0, pj, pi, pn, n_tile * (p.bn / 32));   // the tile's kernel rows
                        } else if (PIECES) {   // both operands
                            const int aw = p.swap ? pj : xw, ah = p.swap ? pi : xh, bw = p.swap ? xw : pj, bh = p.swap ? xh : pi;
                            for (int i = 0; i < a_pieces; ++i)
                                tma_load_4d(a_dst + i * kPieceBytes, &map_a, fb, m_tile * BM + 32 * i, aw, ah, pn);
                            for (int i = 0; i < b_pieces; ++i)
                                tma_load_4d(b_dst + i * kPieceBytes, &map_b, fb, n_tile * p.bn + 32 * i, bw, bh, pn);
                        } else if (!p.swap) {   // A: x (rows c), B: dy (cols o)
                            tma_load_5d(a_dst, &map_a, fb, 0, xw, xh, pn, m_tile * (BM / 32));
                            if constexpr (MT > 1) tma_load_5d(a_dst + A_STAGE_BYTES / MT, &map_a, fb, 0, xw + ow1, xh + oh1, pn, 0);
                            if constexpr (MT > 2) {
                                tma_load_5d(a_dst + 2 * (A_STAGE_BYTES / MT), &map_a, fb, 0, xw + ow2, xh + oh2, pn, 0);
                                tma_load_5d(a_dst + 3 * (A_STAGE_BYTES / MT), &map_a, fb, 0, xw + ow3, xh + oh3, pn, 0);
                            }
                            tma_load_5d(b_dst, &map_b, fb, 0, pj, pi, pn, n_tile * (p.bn / 32));
                        } else {         // A: dy (rows o), B: x (cols c)
                            tma_load_5d(a_dst, &map_a, fb, 0, pj, pi, pn, m_tile * (BM / 32));
                            tma_load_5d(b_dst, &map_b, fb, 0, xw, xh, pn, n_tile * (p.bn / 32));
                        }
                    }
                }
                }
                // on to this warp's next stage
#pragma unroll
                for (int i = 0; i < W; ++i) advance();
                if ((s += W) >= p.stages) { s -= p.stages; phase ^= 1u; }
            }
        }
    } else if (warp == 1 || (W == 2 && warp == 3)) {
        // ===== MMA issuer =====
        {
            const int a_mn = (MODE == MODE_DK && !X3) ? 1 : 0;
            const int b_mn = (MODE == MODE_DX) ? 0 : 1;
            const uint32_t idesc = make_idesc(a_mn, b_mn, p.bn, BM);
            // K-major tile: rows of 128 B, 8-row groups 1024 B apart (stride offset); one MMA (K = 8)
            // consumes 32 B of each row.
            // MN-major tile: [32-channel chunk][k row][128 B]: chunks 4096 B apart (leading offset), the
            // 32-byte-chunk swizzle repeats every 4 k rows, so 4-row groups are 512 B apart (stride
            // offset); one MMA consumes 8 k rows = 1024 B.
            const uint32_t a_lbo = a_mn ? 4096u : 16u, b_lbo = b_mn ? 4096u : 16u;
            const uint32_t a_sbo = a_mn ? 512u : 1024u, b_sbo = b_mn ? 512u : 1024u;
            const uint32_t a_lay = a_mn ? kLayoutSw128Base32 : kLayoutSw128;
            const uint32_t b_lay = b_mn ? kLayoutSw128Base32 : kLayoutSw128;
            const uint32_t a_step = a_mn ? 1024u : 32u, b_step = b_mn ? 1024u : 32u;
            // descriptors of stage 0; a stage further on only changes the 14-bit start-address field
            const uint64_t adesc0 = make_smem_desc(a_base, a_lbo, a_sbo, a_lay);
            const uint64_t bdesc0 = make_smem_desc(b_base, b_lbo, b_sbo, b_lay);
            const uint32_t a_stage16 = A_STAGE_BYTES >> 4, b_stage16 = (uint32_t)b_stage_bytes >> 4;
            const uint32_t tmem_w = tmem_d + (uint32_t)(walker * p.bn);   // kDual: the accumulator of this warp's stages
            int s = walker;
            uint32_t phase = 0;
            {
            for (int it = walker; it < nq; it += W) {
                if (!mbar_wait_warp(full_bar + 8u * s, phase, 1, it, wait_limit)) break;
                if (X3 && !mbar_wait_warp(resid_bar + 8u * s, phase, 3, it, wait_limit)) break;   // (implies full_bar)
                // a new block starts from zero once the epilogue warps have taken the last one over
                const int block = it / kX3Block;
                const bool block_start = X3 && it % kX3Block == 0;
                const int buf = block & (x3_mains - 1);
                if (block_start && block >= x3_mains &&
                    !mbar_wait_warp(promo_empty_bar + 8u * buf, (uint32_t)((block >> (x3_mains - 1)) - 1) & 1u, 6, it, wait_limit))
                    break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (elect_one()) {
                TC_TRACE(1024 + it);
                if (TC_DEBUG_BIT(1)) {   // timing experiment: no MMA, the stage is released at once
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty_bar + 8u * s) : "memory");
                } else {
                    const uint64_t adesc = adesc0 + (uint64_t)(s * a_stage16);
                    const uint64_t bdesc = bdesc0 + (uint64_t)(s * b_stage16);
                    if (X3) {
                        // a*b ~ a_hi*b_lo + a_lo*b_hi + a_hi*b_hi, the small terms first; the tensor core
                        // reads the TF32 part (top 19 bits) of whatever fp32 word it is given
                        const uint32_t ahi = tmem_d + (uint32_t)(x3_a0 + 64 * (it & x3_slot_mask)), alo = ahi + 32u;
                        const uint32_t d_main = tmem_d + (uint32_t)(buf * p.bn), d_small = tmem_d + (uint32_t)(x3_mains * p.bn);
                        const uint64_t bres = bdesc0 + (uint64_t)((bs_base - b_base) >> 4) + (uint64_t)((uint32_t)(it & x3_bslot_mask) * b_stage16);
#pragma unroll
                        for (int kk = 0; kk < BK / 8; ++kk) {
                            const uint64_t kb = (uint64_t)(kk * (b_step >> 4));
                            tcgen05_mma_tf32_ts(d_small, ahi + 8u * kk, bres + kb, idesc, (it > 0 || kk > 0) ? 1u : 0u);
                            tcgen05_mma_tf32_ts(d_small, alo + 8u * kk, bdesc + kb, idesc, 1u);
                            tcgen05_mma_tf32_ts(d_main, ahi + 8u * kk, bdesc + kb, idesc, (!block_start || kk > 0) ? 1u : 0u);
                        }
                    } else {
#pragma unroll
                        for (int kk = 0; kk < BK / 8; ++kk)
                            tcgen05_mma_tf32(tmem_w, adesc + (uint64_t)(kk * (a_step >> 4)), bdesc + (uint64_t)(kk * (b_step >> 4)),
                                             idesc, (it >= W || kk > 0) ? 1u : 0u);
                    }
                    tcgen05_commit(empty_bar + 8u * s);  // frees the stage once these MMAs have read it
                    if (X3 && it % kX3Block == kX3Block - 1 && it + 1 < nq) tcgen05_commit(promo_full_bar + 8u * buf);
                }
                TC_TRACE(2048 + it);
                }
                if ((s += W) >= p.stages) { s -= p.stages; phase ^= 1u; }
            }
            if (elect_one()) tcgen05_commit(tmem_full_bar);   // accumulator complete (or abandoned)
            }
        }
    }
    __syncwarp();
    // how the epilogue threads walk the (row, quad) items of an unpartitioned tile: the first, and the step of EPI items
    int item_r = 0, item_q = 0, step_r = 0, step_q = 0;
    if (warp >= 2) {
        // ===== epilogue, part 1 (warps 2..5; TMEM lane quadrant = warp % 4; thread = accumulator row) =====
        const int qpr = p.bn >> 2;
        item_r = (int)(threadIdx.x - 64) / qpr; item_q = (int)(threadIdx.x - 64) - item_r * qpr;
        step_r = EPI / qpr; step_q = EPI - step_r * qpr;
        pdl_enter();
        const int quad = warp & 3;
        const int row = quad * 32 + lane;
        // where does this accumulator row go?  (worked out while the main loop is still running)
        bool row_valid = false;
        unsigned long long row_off = 0;   // element offset of column 0 of this row
        if (MODE == MODE_FWD) {
            const int tw = row % p.TW, th = (row / p.TW) % p.TH, tn = row / (p.TW * p.TH);
            const int n = n0 + tn, i = i0 + th, j = j0 + tw;
            row_valid = tn < p.TN && n < p.N && i < p.Ho && j < p.Wo;
            row_off = (((unsigned long long)n * p.Ho + i) * p.Wo + j) * p.O + ch0;
            if (p.planes) row_off = (((unsigned long long)n * p.Ho + i) * p.Wo + j) * 4ull;
        } else if (MODE == MODE_DX) {
            const int tw = row % p.TW, th = (row / p.TW) % p.TH, tn = row / (p.TW * p.TH);
            const int n = n0 + tn, h = p.sh * (i0 + th) + ph, w = p.sw * (j0 + tw) + pw;
            row_valid = tn < p.TN && n < p.N && h < p.H && w < p.W;
            row_off = (((unsigned long long)n * p.H + h) * p.W + w) * p.C + ch0;
        } else {
            const unsigned long long tap_off = (unsigned long long)group * p.C * p.O;
            if (p.narrow) {  // rows o, columns = 32 * kernel row + window slot (kernel column dj = slot / 4, channel = slot % 4)
                const int o = m_tile * BM + row;
                row_valid = o < p.O;
                row_off = o;
            } else if (!p.swap) {   // rows c, columns o
                const int t = row / (BM / MT), c = m_tile * BM + row - t * (BM / MT), tap = group * MT + t;
                row_valid = c < p.C && tap < p.KH * p.KW;
                row_off = ((unsigned long long)tap * p.C + c) * p.O + ch0;
            } else {         // rows o, columns c
                const int o = m_tile * BM + row;
                row_valid = o < p.O;
                row_off = tap_off + (unsigned long long)ch0 * p.O + o;
            }
        }
        if constexpr (X3) {
            // ===== 3xTF32: these warps take the landed stages apart, the groups of four in turn =====
            // residual = value - (value with the low 13 mantissa bits cleared).  A: thread = row, values and residuals to
            // the stage's TMEM columns.  B: element-wise on the raw bytes of the stage, so the swizzled layout carries
            // over unchanged.
            // Everything but the stores to TMEM is done before the slot is free, so that little stands between the MMAs that
            // free it and those that read it next; B first, while the registers of A's values can hold eight of its words in flight.
            const int group = (warp - 2) >> 2, tid_r = (threadIdx.x - 64) & 127;
            int turn = 0;
            const int b_q = b_stage_bytes / 16;   // 16-byte words of a B tile
            const int blocks = (nq + kX3Block - 1) / kX3Block;
            int taken = 0;                        // blocks taken over so far
            int s = 0;
            uint32_t phase = 0;
            // the MMAs of the stage n before this one have completed (it was released)
            auto mma_done = [&](int n, int it) {
                if (it < n) return true;
                const bool wrap = s < n;
                const int j = wrap ? s - n + p.stages : s - n;
                return __all_sync(0xffffffffu, mbar_wait(empty_bar + 8u * j, wrap ? phase ^ 1u : phase, 8, it, wait_limit)) != 0;
            };
            for (int it = 0; it < nq; ++it) {
                if (turn == group) {
                    // A wait by parity passes at once on the phase before the last, so a group has to know that the load one round of
                    // the ring earlier has landed.  With as many stages as groups that was its own stage, with two more it is one
                    // whose MMAs it has seen done; with one more it looks at the stage's release first (finish_plan)
                    if (KIND == kX3Wide && !mma_done(p.stages, it)) break;
                    if (!__all_sync(0xffffffffu, mbar_wait(full_bar + 8u * s, phase, 4, it, wait_limit))) break;
                    if (!mma_done(p.x3_bslots, it)) break;
                    const float4* bsrc = reinterpret_cast<const float4*>(smem_raw + (b_base + (uint32_t)s * b_stage_bytes - smem_u32(smem_raw)));
                    float4* bdst = reinterpret_cast<float4*>(smem_raw + (bs_base + (uint32_t)(it & x3_bslot_mask) * b_stage_bytes - smem_u32(smem_raw)));
#pragma unroll 8
                    for (int i = tid_r; i < b_q; i += 128) bdst[i] = tf32_residual(bsrc[i]);
                    const uint8_t* asrc = smem_raw + (a_base + (uint32_t)s * A_STAGE_BYTES - smem_u32(smem_raw));
                    float v[32];
                    if (MODE != MODE_DK) {   // K-major: the row's 128 bytes, 16-byte chunk j at j ^ (row & 7)
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const float4 t = *reinterpret_cast<const float4*>(asrc + row * 128 + ((j ^ (row & 7)) << 4));
                            v[4 * j] = t.x; v[4 * j + 1] = t.y; v[4 * j + 2] = t.z; v[4 * j + 3] = t.w;
                        }
                    } else {                 // MN-major: [32-row chunk][k][128 bytes], 32-byte chunk j at j ^ (k & 3)
#pragma unroll
                        for (int k = 0; k < 32; ++k)
                            v[k] = *reinterpret_cast<const float*>(asrc + quad * 4096 + k * 128 + (((lane >> 3) ^ (k & 3)) << 5) + (lane & 7) * 4);
                    }
                    if (!mma_done(p.x3_slots, it)) break;
                    const uint32_t ahi = tmem_d + ((uint32_t)(quad * 32) << 16) + (uint32_t)(x3_a0 + 64 * (it & x3_slot_mask));
                    tmem_st_32x32b_x32(ahi, v);
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = tf32_residual_1(v[j]);
                    tmem_st_32x32b_x32(ahi + 32u, v);
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic-proxy writes -> tensor core reads
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(resid_bar + 8u * s) : "memory");
                }
                if (++turn == G) turn = 0;
                if (++s == p.stages) { s = 0; phase ^= 1u; }
                // a block is taken over once the first two stages of the next one are ready, so that the tensor core finds
                // work right after it
                if (taken + 1 < blocks && it == min((taken + 1) * kX3Block + 1, nq - 1)) {
                    const int buf = taken & (x3_mains - 1);
                    bool got = mbar_wait(promo_full_bar + 8u * buf, (uint32_t)(taken >> (x3_mains - 1)) & 1u, 7, it, wait_limit);
                    got = __all_sync(0xffffffffu, got);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (!got) break;
                    x3_take_over<KIND>(x3_sum, tmem_d + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * p.bn), group, p.bn);
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(promo_empty_bar + 8u * buf) : "memory");
                    ++taken;
                }
            }
        }
        bool ok = mbar_wait(tmem_full_bar, 0, 2, 0, wait_limit);
        ok = __all_sync(0xffffffffu, ok);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (threadIdx.x == 64) TC_TRACE(3074);
        TC_CTA_TRACE(2);
        if (!ok || nq <= 0) row_valid = false;   // nothing trustworthy to store
        // The pipeline stages are idle from here on (every MMA that read them has completed).
        s_rowoff[row] = row_valid ? (long long)row_off : -1;
    }

    // ===== the K partitions of a tile meet =====
    // The S partitions of one tile form a thread-block cluster, which guarantees that they run at the
    // same time and gives them a hardware barrier.  Each partition writes the others' shares of its partial
    // accumulator to scratch (it stays in L2), the cluster meets, and partition j then finishes a 1/S share of
    // the tile: it adds the others' partials to its own in partition order - so the result does not depend
    // on timing - applies the fused chain and writes the final tensor.  (Through distributed shared memory, by
    // stores or by bulk copies that the receiver's barrier counts, it takes as long or longer.)
    // Partials are stored quad-major, [CTA][16-byte column quad][row]: lanes are consecutive rows, so
    // both the partial stores and the loads of the second phase move 512 contiguous bytes per warp.
    // Without partitions the same layout in shared memory (quad pitch QS) is the transposition buffer
    // between "thread = row" (TMEM) and "warp = row segment" (coalesced global stores).
    const int S = p.splits, part = split;
    const bool multi = S > 1;
    const bool finish_here = !p.ext_finish;   // else: partials only, a second kernel adds them
    const int qpr = p.bn >> 2;                // vector path: 16-byte column quads per row,
    const int QPO = p.by_splits.div(qpr + S - 1);   //   quads per share
    const int QS = BM + 1;                    // shared-memory quad pitch in 16-byte units (odd: lanes = quads hit distinct banks)
    const int CL = p.by_splits.div(p.bn + S - 1);   // scalar path: columns per share
    // Vector path: a partition's own share stays in its TMEM, where the second phase reads it again (with two partitions half of
    // what went through L2: 128 -> 256 forward of 64 images 16.9 -> 16.1 us, with the shorter set-up).  3xTF32 has part of it in
    // registers of other threads.
    const bool keep_own = vec && multi && finish_here && !X3;
    const int own_q0 = part * QPO, own_q = keep_own ? QPO : 0;
    float* my_scratch = p.scratch + (size_t)blockIdx.x * BM * p.bn;
    const float* tile_scratch = p.scratch + (size_t)(blockIdx.x - part) * BM * p.bn;
    if (threadIdx.x == 64) TC_TRACE(3000);
    if (warp >= 2) {
        const int quad = warp & 3;
        const int row = quad * 32 + lane;
        // the warps of a lane quadrant (one per group) take the 32-column slabs in turn (3xTF32: unrolled, for the sums of the
        // slabs are registers only if nothing chooses among them at run time: as local memory they cost every launch 3 us, 8 -> 8
        // input gradient 7.1 for 4.2 us)
#pragma unroll (X3 ? SLABS : 1)
        for (int sl = 0; sl < (X3 ? SLABS : 256 / 32); ++sl) {
            const int c0 = ((warp - 2) >> 2) * 32 + sl * 32 * G;
            if (c0 >= p.bn) break;
            uint32_t r[32];
            const uint32_t tquad = tmem_d + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0;
            const uint32_t taddr = tquad + (X3 ? (uint32_t)(((nq > 0 ? (nq - 1) / kX3Block : 0) & (x3_mains - 1)) * p.bn) : 0u);
            const bool full = p.bn - c0 >= 32;   // bn is a multiple of 16: the last slab has 32 or 16 columns
            if (full) tmem_ld_32x32b_x32(taddr, r);
            else tmem_ld_32x32b_x16(taddr, r);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (W == 2 && nq > 1) {   // the odd stages' accumulator
                uint32_t r2[32];
                if (full) tmem_ld_32x32b_x32(tquad + (uint32_t)p.bn, r2);
                else tmem_ld_32x32b_x16(tquad + (uint32_t)p.bn, r2);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int q = 0; q < 32; ++q)
                    if (q < 16 || full) r[q] = __float_as_uint(__fadd_rn(__uint_as_float(r[q]), __uint_as_float(r2[q])));
            }
            if constexpr (X3) {   // add the accumulator of the small terms, then the blocks taken over before
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    if (half == 1 && !full) break;
                    uint32_t r2[32];   // (16 of them)
                    tmem_ld_32x32b_x16(tquad + (uint32_t)(x3_mains * p.bn + 16 * half), r2);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int q = 0; q < 16; ++q)
                        r[16 * half + q] = __float_as_uint(__fadd_rn(__fadd_rn(x3_sum[sl][16 * half + q], __uint_as_float(r[16 * half + q])), __uint_as_float(r2[q])));
                }
            }
            if (vec) {
                if (multi) {
                    float4* d4 = reinterpret_cast<float4*>(my_scratch) + (size_t)(c0 >> 2) * BM + row;
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if ((q < 4 || full) && (unsigned)((c0 >> 2) + q - own_q0) >= (unsigned)own_q)
                            __stcg(d4 + q * BM, make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]),
                                                            __uint_as_float(r[4 * q + 2]), __uint_as_float(r[4 * q + 3])));
                } else {
                    float4* d4 = reinterpret_cast<float4*>(red) + (c0 >> 2) * QS + row;
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (q < 4 || full)
                            d4[q * QS] = make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]),
                                                     __uint_as_float(r[4 * q + 2]), __uint_as_float(r[4 * q + 3]));
                }
            } else {
                // column-major [column][row], in scratch or in shared memory
                float* d1 = (multi ? my_scratch : red) + (size_t)c0 * BM + row;
#pragma unroll
                for (int q = 0; q < 32; ++q)
                    if (q < 16 || full) d1[q * BM] = __uint_as_float(r[q]);
            }
        }
        // no fence here: every thread's partial stores are ordered before its own arrival at the cluster barrier
        // (barrier.cluster.arrive.release / wait.acquire), and before the finish kernel by the kernel boundary
    }
    if (threadIdx.x == 64) TC_TRACE(3001);
    TC_CTA_TRACE(3);
    __syncwarp();
    if (multi && finish_here) cluster_sync_all();
    else if (warp >= 2) asm volatile("bar.sync 1, %0;" ::"n"(EPI) : "memory");
    if (threadIdx.x == 64) TC_TRACE(3002);
    TC_CTA_TRACE(4);

    if (warp >= 2 && finish_here) {
        // ===== this partition's share: sum in partition order, fused chain, stores =====
        const int tid_e = threadIdx.x - 64;
        const EpilogueArgs& e = p.ep;
        if (vec) {
            const bool fused = e.raw_out || e.bias || e.pre_act || e.gate || e.act != DCG_ACT_NONE;
            // multi: thread = row, items = the quads of this share.  single: item = (row, quad) with
            // consecutive lanes on consecutive quads, so a warp stores whole 128-byte row segments.
            const int Qm = min(QPO, qpr - part * QPO);
            const bool by_row = multi || p.planes;               // thread = row (else: lanes walk the quads of a row)
            // by_row: the G threads of a row (tid_e, tid_e + 128, ...) take the quads in turn
            const int my_row = (warp & 3) * 32 + lane, my_half = tid_e >> 7;   // (the rows of this warp's TMEM lanes)
            const int row_quads = multi ? Qm : qpr;              // by_row: quads of this row's share
            const int per_thread = by_row ? (row_quads > my_half ? (row_quads - my_half + G - 1) / G : 0)
                                          : (BM * qpr + EPI - 1) / EPI;   // single: 128 * qpr items over all threads
            const int quad0 = ch0 >> 2;                          // planes: global index of this tile's first quad
            int rr = item_r, q = item_q;
            const long long my_ro = s_rowoff[my_row];
            const float4* red4 = reinterpret_cast<const float4*>(red);
            const float4* ts4 = reinterpret_cast<const float4*>(tile_scratch);
            for (int base = 0; base < per_thread; base += 4) {
                float4 acc[4];
                long long goff[4];
                int cq[4];
                if (by_row) {
                    const float4* src[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const bool in = base + u < per_thread;
                        const int qd = part * QPO + (in ? my_half + G * (base + u) : 0);
                        cq[u] = qd << 2;
                        goff[u] = (!in || my_ro < 0 || cq[u] >= ncols_valid) ? -1
                                  : p.planes ? my_ro + (long long)((unsigned long long)(quad0 + qd) * p.plane_stride)
                                             : my_ro + cq[u];
                        src[u] = (multi ? ts4 + (size_t)qd * BM : red4 + qd * QS) + my_row;
                    }
                    if (!X3 && multi) {   // this partition's own products first, the others' behind them in partition order
                        const uint32_t at = tmem_d + ((uint32_t)((warp & 3) * 32) << 16);
#pragma unroll
                        for (int u = 0; u < 4; ++u) tmem_ld_32x32b_x4(at + (uint32_t)cq[u], acc[u]);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                        if (W == 2 && nq > 1) {   // the odd stages' accumulator
                            float4 odd[4];
#pragma unroll
                            for (int u = 0; u < 4; ++u) tmem_ld_32x32b_x4(at + (uint32_t)(p.bn + cq[u]), odd[u]);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                acc[u].x = __fadd_rn(acc[u].x, odd[u].x); acc[u].y = __fadd_rn(acc[u].y, odd[u].y);
                                acc[u].z = __fadd_rn(acc[u].z, odd[u].z); acc[u].w = __fadd_rn(acc[u].w, odd[u].w);
                            }
                        }
                    } else {
#pragma unroll
                        for (int u = 0; u < 4; ++u) acc[u] = multi ? __ldcg(src[u]) : *src[u];
                    }
#pragma unroll 2
                    for (int i = 1; i < S; ++i) {   // two partitions' loads in flight
                        const int sidx = X3 || i > part ? i : i - 1;
                        float4 v[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) v[u] = __ldcg(src[u] + (size_t)sidx * BM * qpr);
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            acc[u].x = __fadd_rn(acc[u].x, v[u].x); acc[u].y = __fadd_rn(acc[u].y, v[u].y);
                            acc[u].z = __fadd_rn(acc[u].z, v[u].z); acc[u].w = __fadd_rn(acc[u].w, v[u].w);
                        }
                    }
                } else {
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const bool in = base + u < per_thread && rr < BM;
                        cq[u] = q << 2;
                        const long long ro = in ? s_rowoff[rr] : -1;
                        goff[u] = (ro < 0 || cq[u] >= ncols_valid) ? -1 : ro + cq[u];
                        acc[u] = red4[in ? q * QS + rr : 0];
                        rr += step_r; q += step_q;
                        if (q >= qpr) { q -= qpr; ++rr; }
                    }
                }
                if (fused) {
                    // each optional step of the chain runs over the four items at once, so its
                    // test is paid once and the loads of a step are in flight together
                    if (e.raw_out) {
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (goff[u] >= 0) *reinterpret_cast<float4*>(e.raw_out + goff[u]) = acc[u];
                    }
                    if (e.bias) {
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            // (a tile may have more columns than there are channels left)
                            const float4 bv = __ldg(reinterpret_cast<const float4*>(e.bias + ch0 + (cq[u] < ncols_valid ? cq[u] : 0)));
                            acc[u].x = __fadd_rn(acc[u].x, bv.x); acc[u].y = __fadd_rn(acc[u].y, bv.y);
                            acc[u].z = __fadd_rn(acc[u].z, bv.z); acc[u].w = __fadd_rn(acc[u].w, bv.w);
                        }
                    }
                    if (e.pre_act) {
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (goff[u] >= 0) *reinterpret_cast<float4*>(e.pre_act + goff[u]) = acc[u];
                    }
                    act_apply_all(acc, e.act, e.alpha);
                    if (e.gate) {
                        float4 gg[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            gg[u] = goff[u] >= 0 ? __ldg(reinterpret_cast<const float4*>(e.gate + goff[u]))
                                                 : make_float4(0.f, 0.f, 0.f, 0.f);
                        act_grad_apply_all(acc, gg, e.gate_act, e.gate_alpha);
                    }
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (goff[u] >= 0) *reinterpret_cast<float4*>(p.out + goff[u]) = acc[u];
            }
        } else {
            // thread = row; share = every S-th column.  Used where consecutive ROWS are adjacent in
            // memory (DK with the channel roles swapped, narrow-channel DK) and for channel counts
            // that rule out 16-byte stores.
            const int my_row = tid_e & (BM - 1), my_half = tid_e >> 7;   // the G threads of a row take the columns in turn
            const long long ro = s_rowoff[my_row];
            for (int cl0 = 0; G * cl0 + my_half < CL; cl0 += 4) {   // four columns at a time: their loads are in flight together
                float acc[4];
                int cols[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int cl = G * (cl0 + u) + my_half;
                    const int col = cl * S + part;
                    cols[u] = (cl < CL && col < ncols_valid) ? col : -1;
                    const int cc = cols[u] < 0 ? 0 : cols[u];
                    acc[u] = multi ? __ldcg(tile_scratch + (size_t)cc * BM + my_row) : red[cc * BM + my_row];
                }
                if (multi) {
                    for (int sidx = 1; sidx < S; ++sidx) {
                        float v[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            v[u] = __ldcg(tile_scratch + ((size_t)sidx * p.bn + (cols[u] < 0 ? 0 : cols[u])) * BM + my_row);
#pragma unroll
                        for (int u = 0; u < 4; ++u) acc[u] = __fadd_rn(acc[u], v[u]);
                    }
                }
                if (ro < 0) continue;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int col = cols[u];
                    if (col < 0) continue;
                    unsigned long long id = (unsigned long long)ro + (unsigned long long)col * col_stride;
                    if (MODE == MODE_DK && p.narrow) {
                        const int di = (ch0 + col) >> 5, dj = (col & 31) >> 2, c = col & 3;   // slot = 4*dj + channel
                        if (dj >= p.KW || c >= p.C) continue;                          // padding slots
                        id = (unsigned long long)ro + (unsigned long long)((di * p.KW + dj) * p.C + c) * p.O;
                    }
                    // the fused chain only exists for FWD/DX; DK stores raw sums
                    p.out[id] = (MODE == MODE_DK) ? acc[u] : epilogue_apply(e, acc[u], id, ch0 + col);
                }
            }
        }
    }

    if (threadIdx.x == 64) TC_TRACE(3075);
    TC_CTA_TRACE(5);
    // ---- teardown: everyone is done with TMEM before warp 1 releases it --------------------------
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"(tmem_cols) : "memory");
    }
}

}  // namespace
}  // namespace dcg

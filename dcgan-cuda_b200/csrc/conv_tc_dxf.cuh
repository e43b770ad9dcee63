// conv_dxf_kernel: input gradient with all parity classes of a pixel tile in one CTA.  Included by conv_tc.cu only.
#pragma once

namespace dcg {
namespace {

// ---- DX with all parity classes of a pixel tile in one CTA -------------------------------------------
// The parity classes of the input gradient (pix mod stride) read the SAME windows of dy, only paired
// with different kernel taps: class (ph, pw), tap (di, dj) reads dy at pixel offset
// ((ph + pad - di) / s, (pw + pad - dj) / s) of the class grid.  For a 5x5 kernel at stride 2 the 25
// (class, tap) pairs share 9 distinct windows.  conv_tc_kernel<DX> runs every class as a tile of its
// own and so fetches a dy tile from L2 once per tap; with a narrow N tile (64 input channels: A 16 KB
// against B 8 KB per stage) that fetch is two thirds of what the SM has to take in, and taking
// operands in is what bounds the main loop.  This kernel gives one CTA the 128 pixels of ALL classes:
// one accumulator per class (classes x bn <= 512 TMEM columns), each window fetched once and
// multiplied against the weight tiles of every pair that reads it - 9 x 16 KB + 25 x 8 KB per 32
// output channels instead of 25 x 24 KB.  A pipeline stage is one window plus the weight tiles of up to
// `pb` pairs that read it (a window with more pairs takes several stages and is fetched again for
// each).  The windows are ordered so that the classes complete one after the other; the epilogue
// of a finished class (through shared memory of its own, not the stage ring) runs under
// the main loop of the rest.  No K partitions: the planner only picks this kernel when the tiles
// alone fill the GPU.
//
// A load takes about 1750 clocks to land while the chip is busy, so what is in flight paces the short stages: with slots
// sized for the longest one (48 KB) a stage of two pairs took 650 clocks for 277 of MMAs.  The ring is therefore cut into
// units of 16 KB, of which a stage takes the two or three that it needs, and its barriers go by the stage's number.  Issuing
// five loads takes a warp as long as their MMAs take, so two warps load the stages in turn.  The epilogue has 16 warps,
// each of which transposes 32 rows x 16 columns in a patch of its own - no block-wide barrier - and asks for the
// gate before the class is complete.
//
// The accumulators of the classes sit side by side in TMEM, and the weight tiles of a stage are stacked
// in shared memory in the same order, so pairs whose classes are neighbours there are ONE MMA with
// N = count x bn columns.  That matters for narrow tiles: an N = 64 MMA takes as long as an N = 128
// one (measured: the MMA-only time of the 64-channel layer is 1.8 x that of its N = 128 forward), so
// the 25 N = 64 products of a channel chunk become 4 of N = 256, 4 of N = 128 and 1 of N = 64.
struct CfRun {
    unsigned char count, slot; // one MMA over `count` adjacent accumulators, the first at columns slot * bn ...
    unsigned char pair;        // ... with the weight tiles of the stage from this one on
    unsigned char fresh;       // the first contribution to its classes (in the first channel chunk)
};
struct CfWin {
    signed char sy, sx;        // window: dy pixel (i + sy, j + sx) for class pixel (i, j)
    unsigned char n;           // pairs of this stage, in TMEM order
    unsigned char units;       // ring units it takes
    unsigned char runs;        // MMAs per K step
    unsigned char last;        // bit c: class c is complete with this stage (in the last channel chunk)
    unsigned char kh[4], kw[4];
    CfRun run[4];
};
struct CfTable {
    int nwin, ncls;            // stages per channel chunk, parity classes
    int order[4];              // classes in the order in which they complete
    int slot_of_class[4];      // TMEM position of every class
    CfWin win[32];
};
constexpr int kCfUnit = A_STAGE_BYTES;     // ring unit
constexpr int kCfMaxUnits = 16;
constexpr int kCfBars = 16;                // barrier pairs: stage q uses pair q % 16 (every stage takes two units or more: at most 8 in flight)
constexpr int kCfEpi = 512, kCfThreads = 64 + kCfEpi + 32;   // producer, MMA, 16 epilogue warps, second producer
constexpr int kCfPatch = 32 * 16 * 4;      // bytes of an epilogue warp's patch

// The fused chain over four 16-byte items at once: every optional step is tested once.  goff < 0 marks an item that is not
// stored; the bias and the gate values have been loaded ahead.
__device__ __forceinline__ void cf_chain_store4(const EpilogueArgs& e, float* out, float4 (&acc)[4], const long long (&goff)[4],
                                                const float4 (&bias)[4], const float4 (&gate)[4])
{
    if (e.raw_out) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (goff[u] >= 0) *reinterpret_cast<float4*>(e.raw_out + goff[u]) = acc[u];
    }
    if (e.bias) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            acc[u].x = __fadd_rn(acc[u].x, bias[u].x); acc[u].y = __fadd_rn(acc[u].y, bias[u].y);
            acc[u].z = __fadd_rn(acc[u].z, bias[u].z); acc[u].w = __fadd_rn(acc[u].w, bias[u].w);
        }
    }
    if (e.pre_act) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (goff[u] >= 0) *reinterpret_cast<float4*>(e.pre_act + goff[u]) = acc[u];
    }
    act_apply_all(acc, e.act, e.alpha);
    if (e.gate) act_grad_apply_all(acc, gate, e.gate_act, e.gate_alpha);
#pragma unroll
    for (int u = 0; u < 4; ++u)
        if (goff[u] >= 0) *reinterpret_cast<float4*>(out + goff[u]) = acc[u];
}

// The same where nothing was loaded ahead: the loads of the four items (`ch`: their channels) are in flight together.
__device__ __forceinline__ void cf_chain_store4(const EpilogueArgs& e, float* out, float4 (&acc)[4], const long long (&goff)[4],
                                                const int (&ch)[4])
{
    float4 bias[4], gate[4];
    if (e.bias) {
#pragma unroll
        for (int u = 0; u < 4; ++u) bias[u] = __ldg(reinterpret_cast<const float4*>(e.bias + ch[u]));
    }
    if (e.gate) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
            gate[u] = goff[u] >= 0 ? __ldg(reinterpret_cast<const float4*>(e.gate + goff[u])) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    cf_chain_store4(e, out, acc, goff, bias, gate);
}

__global__ void __launch_bounds__(kCfThreads, 1)
conv_dxf_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                const __grid_constant__ Params p, const __grid_constant__ CfTable t)
{
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem0 = smem_u32(smem_raw);
    const uint32_t ring = (smem0 + 1023u) & ~1023u;
    const long long wait_limit = p.wait_cycles;
    const int units = p.stages;                             // ring units
    const uint32_t patch_base = ring + (uint32_t)(units * kCfUnit);
    const uint32_t bar_base = patch_base + (uint32_t)(kCfEpi / 32 * kCfPatch);
    const uint32_t full_bar = bar_base;                     // the stage has landed
    const uint32_t empty_bar = bar_base + 8u * kCfBars;     // the MMAs that read it have completed
    const uint32_t cls_bar = bar_base + 16u * kCfBars;      // accumulator of class c complete
    const uint32_t tmem_slot = cls_bar + 32u;
    uint32_t* tmem_slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (tmem_slot - smem0));

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int ncls = t.ncls, nwin = t.nwin;
    const uint32_t b_bytes = (uint32_t)p.bn * BK * 4;

    if (warp == 0) {   // a lane per barrier
        if (lane < kCfBars) {
            mbar_init(full_bar + 8u * lane, 1);
            mbar_init(empty_bar + 8u * lane, 1);
        }
        if (lane < 4) mbar_init(cls_bar + 8u * lane, 1);
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        __syncwarp();
    }
    int tmem_cols = 32;
    while (tmem_cols < ncls * p.bn) tmem_cols <<= 1;
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // blockIdx.x = pixel tile * n_tiles + channel tile
    int n_tile, m_tile, j0, i0, n0;
    p.by_n_tiles.divmod((int)blockIdx.x, m_tile, n_tile);
    p.by_tiles_w.divmod(m_tile, n0, j0);
    p.by_tiles_h.divmod(n0, n0, i0);
    j0 *= p.TW; i0 *= p.TH; n0 *= p.TN;
    const int ch0 = n_tile * p.bn;
    const int ncols_valid = min(p.bn, p.C - ch0);

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_d = *tmem_slot_ptr;

    if (warp == 0 || warp == 2 + kCfEpi / 32) {
        // ===== TMA producers: for every table entry, for every channel chunk: the window, then its weight tiles =====
        // Both walk all stages, to know where each one lies, and load the even ones or the odd ones.
        const int mine = warp == 0 ? 0 : 1;
        int u = 0, q = 0;
        uint32_t used = 0;                // bit u: unit u has been part of a stage ...
        unsigned long long owner = 0;     // ... four bits per unit: the last such stage's number modulo 16
        auto own = [&](int first, int end, int stage) {
            const unsigned long long mask = (~0ull >> (64 - 4 * (end - first))) << (4 * first);
            owner = (owner & ~mask) | ((0x1111111111111111ull * (unsigned long long)(stage & 15)) & mask);
            used |= ((1u << (end - first)) - 1u) << first;
        };
        bool alive = true;
        pdl_enter();
        for (int w = 0; w < nwin && alive; ++w) {
            const CfWin& wn = t.win[w];
            const int aj = j0 + wn.sx, ai = i0 + wn.sy, np = wn.n, nu = wn.units;
            int kh[4], kw[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) { kh[j] = wn.kh[j]; kw[j] = wn.kw[j]; }
            const uint32_t tx_bytes = (uint32_t)A_STAGE_BYTES + (uint32_t)np * b_bytes;
            for (int chunk = 0; chunk < p.kchunks; ++chunk, ++q) {
                if (u + nu > units) {   // a stage is contiguous; what is left over counts as the last stage's
                    own(u, units, q - 1);
                    u = 0;
                }
                if ((q & 1) == mine) {
                    // stages complete in order: the last unit's owner is the youngest that has to be out of the way
                    const int last = u + nu - 1;
                    if ((used >> last) & 1u) {
                        const int slot = (int)(owner >> (4 * last)) & 15, prev = q - 1 - ((q - 1 - slot) & 15);
                        if (!mbar_wait_warp(empty_bar + 8u * slot, (uint32_t)(prev >> 4) & 1u, 0, q, wait_limit)) { alive = false; break; }
                    }
                    if (elect_one()) {
                        const uint32_t fb = full_bar + 8u * (q & 15);
                        const uint32_t dst = ring + (uint32_t)(u * kCfUnit);
                        mbar_expect_tx(fb, tx_bytes);
                        tma_load_4d(dst, &map_a, fb, chunk * BK, aj, ai, n0);
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            if (j < np) tma_load_4d(dst + (uint32_t)A_STAGE_BYTES + (uint32_t)j * b_bytes, &map_b, fb, chunk * BK, ch0, kw[j], kh[j]);
                    }
                }
                own(u, u + nu, q);
                u += nu;
                if (u == units) u = 0;
            }
        }
    } else if (warp == 1) {
        // ===== MMA issuer =====
        // The MMAs of a table entry are worked out one entry ahead, under MMAs: read when the entry begins, they cost 450
        // clocks per entry.
        const uint64_t desc0 = make_smem_desc(ring, 16u, 1024u, kLayoutSw128);   // K-major, 128-byte rows, 8-row groups 1024 B apart
        const uint32_t b16 = b_bytes >> 4;
        struct Runs {
            uint32_t idesc[4], acc[4], b_off[4], fresh, last;
            int n, units;
        };
        auto fetch = [&](int w) {
            const CfWin& wn = t.win[w];
            Runs r;
            r.n = wn.runs; r.units = wn.units; r.last = wn.last;
            r.fresh = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const CfRun c = wn.run[i];
                r.idesc[i] = make_idesc(0, 0, c.count * p.bn, BM);
                r.acc[i] = tmem_d + (uint32_t)(c.slot * p.bn);
                r.b_off[i] = (uint32_t)(A_STAGE_BYTES >> 4) + (uint32_t)c.pair * b16;
                r.fresh |= (uint32_t)c.fresh << i;
            }
            return r;
        };
        int u = 0, it = 0;
        uint32_t done = 0;
        bool alive = true;
        Runs cur = fetch(0), next = cur;
        for (int w = 0; w < nwin && alive; ++w) {
            for (int chunk = 0; chunk < p.kchunks; ++chunk, ++it) {
                if (u + cur.units > units) u = 0;
                if (!mbar_wait_warp(full_bar + 8u * (it & 15), (uint32_t)(it >> 4) & 1u, 1, it, wait_limit)) { alive = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const bool final_chunk = chunk == p.kchunks - 1;
                if (elect_one()) {
                    const uint64_t adesc = desc0 + (uint64_t)((uint32_t)u * (uint32_t)(kCfUnit >> 4));
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        if (r < cur.n) {   // one MMA per K step over the adjacent accumulators of this run
                            const uint64_t bdesc = adesc + (uint64_t)cur.b_off[r];
                            const bool overwrite = chunk == 0 && ((cur.fresh >> r) & 1u);
#pragma unroll
                            for (int kk = 0; kk < BK / 8; ++kk)
                                tcgen05_mma_tf32(cur.acc[r], adesc + (uint64_t)(kk * 2), bdesc + (uint64_t)(kk * 2), cur.idesc[r],
                                                 (overwrite && kk == 0) ? 0u : 1u);
                        }
                    tcgen05_commit(empty_bar + 8u * (it & 15));
                    if (final_chunk) {
#pragma unroll
                        for (int c = 0; c < 4; ++c)
                            if ((cur.last >> c) & 1u) tcgen05_commit(cls_bar + 8u * c);
                    }
                }
                if (final_chunk) done |= cur.last;
                if (chunk == 0 && w + 1 < nwin) next = fetch(w + 1);
                u += cur.units;
                if (u == units) u = 0;
            }
            cur = next;
        }
        // a pipeline that gave up still releases the epilogue (which stores nothing then)
        if (elect_one())
            for (int c = 0; c < ncls; ++c)
                if (!((done >> c) & 1u)) tcgen05_commit(cls_bar + 8u * c);
    } else {
        // ===== epilogue: classes in completion order, 32 rows x 16 accumulator columns per warp at a time =====
        // Four warps per TMEM lane quadrant take the 16-column pieces of a class in turn.  The patch between "thread = row"
        // and "four lanes = 64 contiguous bytes of a row" holds row r's column quad q at place q ^ ((r >> 1) & 3), which
        // keeps the banks of both sides apart.
        const int quad = warp & 3, piece0 = (warp - 2) >> 2;
        const int row = quad * 32 + lane;
        const int tw = row % p.TW, th = (row / p.TW) % p.TH, tn = row / (p.TW * p.TH);
        const EpilogueArgs& e = p.ep;
        float4* patch = reinterpret_cast<float4*>(smem_raw + (patch_base - smem0) + (warp - 2) * kCfPatch);
        const float* patch1 = reinterpret_cast<const float*>(patch);
        // 16-byte stores need whole column quads in every row; else element by element
        const bool vec = (p.C & 3) == 0 && (ncols_valid & 3) == 0;
        pdl_enter();
        for (int ci = 0; ci < ncls; ++ci) {
            const int cls = t.order[ci];
            const int ph = cls / p.sw, pw = cls % p.sw;
            const int n = n0 + tn, h = p.sh * (i0 + th) + ph, w = p.sw * (j0 + tw) + pw;
            const bool valid = n < p.N && h < p.H && w < p.W;
            const long long my_off = valid ? (long long)((((unsigned long long)n * p.H + h) * p.W + w) * p.C + ch0) : -1;
            bool waited = false, ok = true;
            for (int c0 = piece0 * 16; c0 < p.bn; c0 += 64) {
                const int col = c0 + (lane & 3) * 4;
                long long goff[4];
                float4 gate[4], bias[4];
                if (vec) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const long long ro = __shfl_sync(0xffffffffu, my_off, 8 * u + (lane >> 2));
                        goff[u] = ro < 0 || col >= ncols_valid ? -1 : ro + col;
                    }
                    if (e.bias) {
                        const float4 bv = __ldg(reinterpret_cast<const float4*>(e.bias + ch0 + (col < ncols_valid ? col : 0)));
                        bias[0] = bv; bias[1] = bv; bias[2] = bv; bias[3] = bv;
                    }
                    if (e.gate) {
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            gate[u] = goff[u] >= 0 ? __ldg(reinterpret_cast<const float4*>(e.gate + goff[u])) : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                }
                if (!waited) {
                    ok = __all_sync(0xffffffffu, mbar_wait(cls_bar + 8u * cls, 0, 2, cls, wait_limit));
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    waited = true;
                }
                uint32_t r[32];
                tmem_ld_32x32b_x16(tmem_d + ((uint32_t)(quad * 32) << 16) + (uint32_t)(t.slot_of_class[cls] * p.bn + c0), r);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    patch[lane * 4 + (q ^ ((lane >> 1) & 3))] = make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]),
                                                                             __uint_as_float(r[4 * q + 2]), __uint_as_float(r[4 * q + 3]));
                __syncwarp();
                if (vec) {
                    float4 acc[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int rr = 8 * u + (lane >> 2);
                        acc[u] = patch[rr * 4 + ((lane & 3) ^ ((rr >> 1) & 3))];
                        if (!ok) goff[u] = -1;
                    }
                    cf_chain_store4(e, p.out, acc, goff, bias, gate);
                } else {   // two rows of 16 columns at a time
                    for (int u = 0; u < 16; ++u) {
                        const int rr = 2 * u + (lane >> 4), c = lane & 15;
                        const long long ro = __shfl_sync(0xffffffffu, my_off, rr);
                        if (!ok || ro < 0 || c0 + c >= ncols_valid) continue;
                        const unsigned long long id = (unsigned long long)ro + (unsigned long long)(c0 + c);
                        p.out[id] = epilogue_apply(e, patch1[rr * 16 + (((c >> 2) ^ ((rr >> 1) & 3)) << 2) + (c & 3)], id, ch0 + c0 + c);
                    }
                }
                __syncwarp();
            }
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"(tmem_cols) : "memory");
    }
}

}  // namespace
}  // namespace dcg

// conv_tc_walk_kernel: forward and input gradient of layers with more tiles than SMs, as persistent CTAs.  Included by conv_tc.cu only.
#pragma once

namespace dcg {
namespace {

// ---- more tiles than SMs ------------------------------------------------------------------------------
// A stage takes about 1500 clocks from its load to its release, so what paces the main loop is how many are in flight: seven
// stages of 128 columns go through at 290 clocks each, two CTAs of three stages that share an SM at 500.  Those two hide one's
// epilogue behind the other's stages; here one CTA per SM does so by itself.  It walks tiles blockIdx.x, blockIdx.x + gridDim.x,
// ... with the whole of shared memory for its ring, which goes on from one tile to the next, and two accumulators in TMEM: a
// tile's epilogue, through a patch of its own per warp (as in conv_dxf_kernel), runs under the next tile's products.  Two warps
// load the stages in turn.
// Against two CTAs per SM: 1 x 1, 64 -> 192, 16 images of 96 x 96 forward 47.8 -> 31.2 us, input gradient 34.1 -> 25.3; 3 x 3, 96 -> 160,
// 13 images of 75 x 51 32.6 -> 24.1 and 35.4 -> 28.2; 64 -> 128 of 512 images 106.4 -> 95.8, of 128 images 27.3 -> 26.7.
constexpr int kWalkEpi = 512, kWalkThreads = 64 + kWalkEpi + 32;   // producer, MMA, 16 epilogue warps, second producer
constexpr int kWalkPatch = 32 * 16 * 4;   // bytes of an epilogue warp's patch

__host__ __device__ constexpr size_t walk_smem(int stages, int bn)
{
    return 1024 + (size_t)stages * (A_STAGE_BYTES + bn * BK * 4) + kWalkEpi / 32 * kWalkPatch + 16 * stages + 64;
}

// PIECES (forward): ragged channel counts, B in loads of 32 columns, of which those that exist.
template <int MODE, bool PIECES = false>
__global__ void __launch_bounds__(kWalkThreads, 1)
conv_tc_walk_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                    const __grid_constant__ Params p, const int tiles)
{
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem0 = smem_u32(smem_raw);
    const uint32_t a_base = (smem0 + 1023u) & ~1023u;
    const uint32_t b_stage = (uint32_t)p.bn * BK * 4;
    const uint32_t b_base = a_base + (uint32_t)p.stages * A_STAGE_BYTES;
    const uint32_t patch_base = b_base + (uint32_t)p.stages * b_stage;
    const uint32_t full_bar = patch_base + (uint32_t)(kWalkEpi / 32 * kWalkPatch);
    const uint32_t empty_bar = full_bar + 8u * p.stages;
    const uint32_t acc_full = empty_bar + 8u * p.stages, acc_empty = acc_full + 16u;   // [2] accumulator complete / drained
    const uint32_t tmem_slot = acc_empty + 16u;
    uint32_t* tmem_slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (tmem_slot - smem0));
    const long long wait_limit = p.wait_cycles;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

    if (warp == 0) {   // a lane per barrier
        if (lane < p.stages) {
            mbar_init(full_bar + 8u * lane, 1);
            mbar_init(empty_bar + 8u * lane, 1);
        }
        if (lane < 2) {
            mbar_init(acc_full + 8u * lane, 1);
            mbar_init(acc_empty + 8u * lane, kWalkEpi / 32);
        }
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        __syncwarp();
    }
    int tmem_cols = 32;
    while (tmem_cols < 2 * p.bn) tmem_cols <<= 1;
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_d = *tmem_slot_ptr;

    // A tile: its channels, first pixel and - input gradient - parity class, in the order of conv_tc_kernel's CTAs (the classes
    // with the most taps first).
    struct Tile {
        int n_tile, j0, i0, n0, ph, pw, rh, rw, eh, ew, taps_w, nq;
    };
    auto decode = [&](int tile) {
        Tile t{};
        int rem, m_tile, group;
        p.by_n_tiles.divmod(tile, rem, t.n_tile);
        p.by_m_count.divmod(rem, group, m_tile);
        p.by_tiles_w.divmod(m_tile, t.n0, t.j0);
        p.by_tiles_h.divmod(t.n0, t.n0, t.i0);
        t.j0 *= p.TW; t.i0 *= p.TH; t.n0 *= p.TN;
        if (MODE == MODE_DX) {
            p.by_sw.divmod(group, t.rh, t.rw);
            t.ph = t.rh - p.pt_mod; if (t.ph < 0) t.ph += p.sh;
            t.pw = t.rw - p.pl_mod; if (t.pw < 0) t.pw += p.sw;
            t.eh = p.by_sh.div(t.ph + p.pt); t.ew = p.by_sw.div(t.pw + p.pl);
            const int taps_h = t.rh < p.KH ? p.by_sh.div(p.KH - t.rh + p.sh - 1) : 0;
            t.taps_w = t.rw < p.KW ? p.by_sw.div(p.KW - t.rw + p.sw - 1) : 0;
            t.nq = taps_h * t.taps_w * p.kchunks;
        } else {
            t.taps_w = p.KW;
            t.nq = p.KH * p.KW * p.kchunks;
        }
        return t;
    };

    if (warp == 0 || warp == 2 + kWalkEpi / 32) {
        // ===== TMA producers: both walk all stages, one loads the even and one the odd ones =====
        const int mine = warp == 0 ? 0 : 1;
        const uint32_t a_bytes = (uint32_t)(p.TW * p.TH * p.TN * BK * 4);
        int s = 0, it = 0;
        uint32_t phase = 0;
        bool alive = true;
        pdl_enter();
        for (int tile = blockIdx.x; tile < tiles && alive; tile += gridDim.x) {
            const Tile t = decode(tile);
            const int pieces = PIECES ? min(p.bn >> 5, (p.b_ch - t.n_tile * p.bn + 31) >> 5) : 0;
            int chunk = 0, tap = 0, di = 0, dj = 0;
            for (int q = 0; q < t.nq; ++q, ++it) {
                if ((it & 1) == mine) {
                    if (!mbar_wait_warp(empty_bar + 8u * s, phase ^ 1u, 0, it, wait_limit)) { alive = false; break; }
                    if (it != p.skip_stage && elect_one()) {
                        const uint32_t fb = full_bar + 8u * s;
                        const uint32_t a_dst = a_base + (uint32_t)s * A_STAGE_BYTES, b_dst = b_base + (uint32_t)s * b_stage;
                        mbar_expect_tx(fb, a_bytes + (PIECES ? (uint32_t)pieces * kPieceBytes : b_stage));
                        if (MODE == MODE_FWD) {
                            tma_load_4d(a_dst, &map_a, fb, chunk * BK, p.sw * t.j0 + dj - p.pl, p.sh * t.i0 + di - p.pt, t.n0);
                            if constexpr (PIECES) {
                                for (int i = 0; i < pieces; ++i)
                                    tma_load_4d(b_dst + i * kPieceBytes, &map_b, fb, t.n_tile * p.bn + 32 * i, chunk * BK, tap, 0);
                            } else {
                                tma_load_4d(b_dst, &map_b, fb, 0, chunk * BK, tap, t.n_tile * (p.bn / 32));
                            }
                        } else {   // (di, dj) count the taps of this parity class: kernel tap (rh + sh*di, rw + sw*dj)
                            tma_load_4d(a_dst, &map_a, fb, chunk * BK, t.j0 + t.ew - dj, t.i0 + t.eh - di, t.n0);
                            tma_load_4d(b_dst, &map_b, fb, chunk * BK, t.n_tile * p.bn, t.rw + p.sw * dj, t.rh + p.sh * di);
                        }
                    }
                }
                if (++chunk == p.kchunks) {
                    chunk = 0; ++tap;
                    if (++dj == t.taps_w) { dj = 0; ++di; }
                }
                if (++s == p.stages) { s = 0; phase ^= 1u; }
            }
        }
    } else if (warp == 1) {
        // ===== MMA issuer: A K-major, B MN-major (forward) or K-major; descriptors as in conv_tc_kernel =====
        const int b_mn = MODE == MODE_DX ? 0 : 1;
        const uint32_t idesc = make_idesc(0, b_mn, p.bn, BM);
        const uint64_t adesc0 = make_smem_desc(a_base, 16u, 1024u, kLayoutSw128);
        const uint64_t bdesc0 = b_mn ? make_smem_desc(b_base, 4096u, 512u, kLayoutSw128Base32) : make_smem_desc(b_base, 16u, 1024u, kLayoutSw128);
        const uint32_t b_step = b_mn ? 64u : 2u;
        int s = 0, it = 0, n = 0;
        uint32_t phase = 0;
        bool alive = true;
        for (int tile = blockIdx.x; tile < tiles && alive; tile += gridDim.x, ++n) {
            const int nq = decode(tile).nq, buf = n & 1;
            // the epilogue has drained this accumulator's previous tile (first use: passes at once)
            alive = mbar_wait_warp(acc_empty + 8u * buf, ((uint32_t)(n >> 1) & 1u) ^ 1u, 1, it, wait_limit);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t acc = tmem_d + (uint32_t)(buf * p.bn);
            for (int q = 0; q < nq && alive; ++q, ++it) {
                if (!mbar_wait_warp(full_bar + 8u * s, phase, 1, it, wait_limit)) { alive = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (elect_one()) {
                    const uint64_t adesc = adesc0 + (uint64_t)((uint32_t)s * (A_STAGE_BYTES >> 4)), bdesc = bdesc0 + (uint64_t)((uint32_t)s * (b_stage >> 4));
#pragma unroll
                    for (int kk = 0; kk < BK / 8; ++kk)
                        tcgen05_mma_tf32(acc, adesc + (uint64_t)(kk * 2), bdesc + (uint64_t)(kk * b_step), idesc, (q > 0 || kk > 0) ? 1u : 0u);
                    tcgen05_commit(empty_bar + 8u * s);
                }
                if (++s == p.stages) { s = 0; phase ^= 1u; }
            }
            if (elect_one()) tcgen05_commit(acc_full + 8u * buf);   // complete, or abandoned
        }
    } else {
        // ===== epilogue: 32 rows x 16 accumulator columns per warp at a time, as in conv_dxf_kernel =====
        const int quad = warp & 3, piece0 = (warp - 2) >> 2;
        const int row = quad * 32 + lane;
        const int tw = row % p.TW, th = (row / p.TW) % p.TH, tn = row / (p.TW * p.TH);
        const EpilogueArgs& e = p.ep;
        float4* patch = reinterpret_cast<float4*>(smem_raw + (patch_base - smem0) + (warp - 2) * kWalkPatch);
        const float* patch1 = reinterpret_cast<const float*>(patch);
        const int channels = MODE == MODE_DX ? p.C : p.O;
        pdl_enter();
        int n_it = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++n_it) {
            const Tile t = decode(tile);
            const int buf = n_it & 1, ch0 = t.n_tile * p.bn, ncols_valid = min(p.bn, channels - ch0);
            const bool vec = (channels & 3) == 0;   // (a tile's valid columns are then whole quads, too)
            const int n = t.n0 + tn;
            long long my_off = -1;
            if (MODE == MODE_FWD) {
                const int i = t.i0 + th, j = t.j0 + tw;
                if (tn < p.TN && n < p.N && i < p.Ho && j < p.Wo) my_off = (long long)((((unsigned long long)n * p.Ho + i) * p.Wo + j) * p.O + ch0);
            } else {
                const int h = p.sh * (t.i0 + th) + t.ph, w = p.sw * (t.j0 + tw) + t.pw;
                if (tn < p.TN && n < p.N && h < p.H && w < p.W) my_off = (long long)((((unsigned long long)n * p.H + h) * p.W + w) * p.C + ch0);
            }
            bool waited = false;
            auto hand_back = [&] {
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acc_empty + 8u * buf) : "memory");
            };
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
                    ok = ok && mbar_wait_warp(acc_full + 8u * buf, (uint32_t)(n_it >> 1) & 1u, 2, n_it, wait_limit);   // (waits in vain once at most)
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    waited = true;
                }
                uint32_t r[32];
                tmem_ld_32x32b_x16(tmem_d + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * p.bn + c0), r);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (c0 + 64 >= p.bn) hand_back();   // this warp's last read of the accumulator
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
            if (!waited) {   // a warp without columns still waits for the tile and hands it back
                ok = ok && mbar_wait_warp(acc_full + 8u * buf, (uint32_t)(n_it >> 1) & 1u, 2, n_it, wait_limit);
                hand_back();
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

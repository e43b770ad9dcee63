// conv_dx3_kernel: input gradient of a <= 4-channel layer, GEMM and gather in one persistent kernel.  Included by
// conv_tc.cu only.
#pragma once

namespace dcg {
namespace {

// ---- input gradient of a <= 4-channel layer: GEMM and gather in one persistent kernel -----------------
// dx[n, h, w, c] = sum over the taps of matching parity of ycol[tap][n, i, j][c], where ycol = dy x k^T is
// the plain GEMM of every dy pixel against all taps (N = 4 columns per tap).  Written to memory, ycol is
// 100 floats per dy pixel - 26 MB at batch 64 for a 3 MB result - and the gather is a second launch.
// Here a CTA owns 2R output rows of one image: it runs the GEMM for the R + 2 dy rows that contribute to
// them (two 128-pixel M tiles = 8 rows of 32 pixels, so the rows at the seams are computed twice), parks
// the products in shared memory as [tap][dy pixel][4] and gathers its own output pixels from there, fused
// chain included.  Nothing but dy, the weights and dx touches memory, and it is one launch.  Persistent:
// a CTA walks tiles blockIdx.x, blockIdx.x + gridDim.x, ...; the weights stay resident (read from k
// itself, K-major rows 4 * tap + c), the dy tiles of the next tile stream in and its MMAs run while this
// tile is being gathered (one TMEM accumulator per M tile, handed back as soon as it is in shared memory).
struct Dx3Args {
    int R;            // dy rows owned per tile (2R output rows)
    int mts;          // M tiles (four dy rows) that hold the rows contributing to them: 1 or 2
    int lo;           // first dy row a tile needs, relative to its first owned row (<= 0)
    int tiles_per_img, tiles;
    FastDiv by_tiles_per_img;
};
constexpr int kDx3Rows = 8;                               // dy rows per tile (two M tiles of 4 rows x 32 pixels)
constexpr int kDx3Stages = 4;
constexpr int kDx3Epi = 512;                              // epilogue threads: 16 warps, four per TMEM lane quadrant (one 32-column slab each)
constexpr int kDx3Threads = 64 + kDx3Epi;
constexpr int kDx3YcolBytes = 32 * kDx3Rows * 32 * 16;    // up to 32 taps x 256 dy pixels x 4 floats

// The tile's own output pixels from the products of its dy rows.  Any kernel size: consecutive threads take consecutive pixels.
__device__ __forceinline__ void dx3_gather(const Params& p, const Dx3Args& g, const float4* ycol, int n, int t, bool ok, int tid)
{
    const EpilogueArgs& e = p.ep;
    const int W = p.W, own = 2 * g.R * W, i_base = g.R * t + g.lo;
    for (int px = tid; px < own; px += kDx3Epi) {
        const int hl = px / W, w = px - hl * W;
        const int h = 2 * g.R * t + hl;
        if (h >= p.H || !ok) continue;
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        const int di0 = (h + p.pt) & 1, dj0 = (w + p.pl) & 1;   // kernel rows / columns of matching parity, ascending
        for (int di = di0; di < p.KH; di += 2) {
            const int i = (h + p.pt - di) >> 1;
            if (h + p.pt - di < 0 || i >= p.Ho) continue;
            const int rl = i - i_base;
            for (int dj = dj0; dj < p.KW; dj += 2) {
                const int j = (w + p.pl - dj) >> 1;
                if (w + p.pl - dj < 0 || j >= p.Wo) continue;
                const float4 v = ycol[((di * p.KW + dj) * kDx3Rows + rl) * 32 + j];
                acc[0] = __fadd_rn(acc[0], v.x); acc[1] = __fadd_rn(acc[1], v.y);
                acc[2] = __fadd_rn(acc[2], v.z); acc[3] = __fadd_rn(acc[3], v.w);
            }
        }
        const size_t pix = ((size_t)n * p.H + h) * W + w;
        for (int c = 0; c < p.C; ++c) {
            const size_t idx = pix * p.C + c;
            p.out[idx] = epilogue_apply(e, acc[c], idx, c);
        }
    }
}

// Known kernel size: a lane takes the two neighbouring pixels 2j and 2j + 1 of an output row and a warp a row, so that all of
// a warp's reads of a tap are one contiguous line, a tap is read by those pixels only that it contributes to, and of an RGB
// image a lane stores six floats in a row.  (Pixel by pixel, with the taps chosen by the lane's parity and the bias, the gate and
// the stores handled channel by channel, a tile took 4.3 us: 64 -> 3 input gradient of 256 images 42.6 -> 25.9 us, of 64 images
// 14.5 -> 10.2.)
template <int KH, int KW>
__device__ __forceinline__ void dx3_gather_pairs(const Params& p, const Dx3Args& g, const float4* ycol, int n, int t, bool ok, int warp, int lane)
{
    constexpr int TH = (KH + 1) / 2, TW = (KW + 1) / 2;
    const EpilogueArgs& e = p.ep;
    const int pairs = (p.W + 1) >> 1, chunks = (pairs + 31) >> 5;
    const bool rgb = p.C == 3 && (p.W & 1) == 0 && !e.raw_out && !e.pre_act &&
                     ((reinterpret_cast<uintptr_t>(p.out) | reinterpret_cast<uintptr_t>(e.gate)) & 7u) == 0;
    for (int item = warp; item < 2 * g.R * chunks; item += kDx3Epi / 32) {
        const int line = chunks == 1 ? item : item / chunks, jj = (item - line * chunks) * 32 + lane;
        const int r = line >> 1, ph = line & 1;
        const int h = 2 * (g.R * t + r) + ph, w = 2 * jj;
        if (h >= p.H || jj >= pairs || !ok) continue;
        const size_t pix = ((size_t)n * p.H + h) * p.W + w;
        float2 gate[3];
        if (rgb && e.gate) {
#pragma unroll
            for (int q = 0; q < 3; ++q) gate[q] = __ldg(reinterpret_cast<const float2*>(e.gate + pix * 3) + q);
        }
        // kernel rows and columns of matching parity, ascending: row di0 + 2a reads dy row i0 - a, column dj0 + 2b dy column j0 - b
        const int di0 = (ph + p.pt) & 1, i0 = g.R * t + r + ((ph + p.pt - di0) >> 1), rl0 = i0 - (g.R * t + g.lo);
        float acc[2][4];
#pragma unroll
        for (int pw = 0; pw < 2; ++pw) {
            const int dj0 = (pw + p.pl) & 1, j0 = jj + ((pw + p.pl - dj0) >> 1);
            float4 v[TH * TW];
#pragma unroll
            for (int a = 0; a < TH; ++a) {
                const int di = di0 + 2 * a;
                const bool row_ok = di < KH && i0 - a >= 0 && i0 - a < p.Ho;
#pragma unroll
                for (int b = 0; b < TW; ++b) {
                    const int dj = dj0 + 2 * b;
                    const bool in = row_ok && dj < KW && j0 - b >= 0 && j0 - b < p.Wo;
                    v[a * TW + b] = in ? ycol[((di * KW + dj) * kDx3Rows + rl0 - a) * 32 + j0 - b] : make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
            acc[pw][0] = acc[pw][1] = acc[pw][2] = acc[pw][3] = 0.f;
#pragma unroll
            for (int q = 0; q < TH * TW; ++q) {
                acc[pw][0] = __fadd_rn(acc[pw][0], v[q].x); acc[pw][1] = __fadd_rn(acc[pw][1], v[q].y);
                acc[pw][2] = __fadd_rn(acc[pw][2], v[q].z); acc[pw][3] = __fadd_rn(acc[pw][3], v[q].w);
            }
        }
        if (rgb) {
            float f[6];
#pragma unroll
            for (int q = 0; q < 6; ++q) f[q] = acc[q / 3][q % 3];
            if (e.bias) {
                const float b0 = __ldg(e.bias), b1 = __ldg(e.bias + 1), b2 = __ldg(e.bias + 2);
#pragma unroll
                for (int q = 0; q < 6; ++q) f[q] = __fadd_rn(f[q], q % 3 == 0 ? b0 : q % 3 == 1 ? b1 : b2);
            }
            act_apply_all(f, e.act, e.alpha);
            if (e.gate) {
                const float gv[6] = {gate[0].x, gate[0].y, gate[1].x, gate[1].y, gate[2].x, gate[2].y};
                act_grad_apply_all(f, gv, e.gate_act, e.gate_alpha);
            }
            float2* o = reinterpret_cast<float2*>(p.out + pix * 3);
#pragma unroll
            for (int q = 0; q < 3; ++q) o[q] = make_float2(f[2 * q], f[2 * q + 1]);
        } else {
#pragma unroll
            for (int pw = 0; pw < 2; ++pw) {
                if (w + pw >= p.W) break;
                for (int c = 0; c < p.C; ++c) {
                    const size_t idx = (pix + pw) * p.C + c;
                    p.out[idx] = epilogue_apply(e, c == 0 ? acc[pw][0] : c == 1 ? acc[pw][1] : c == 2 ? acc[pw][2] : acc[pw][3], idx, c);
                }
            }
        }
    }
}

template <int KH_, int KW_>   // 5, 5: tap loops unrolled, all loads of a pixel in flight; 0, 0: any kernel size
__global__ void __launch_bounds__(kDx3Threads, 1)
conv_dx3_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                const __grid_constant__ Params p, const __grid_constant__ Dx3Args g)
{
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem0 = smem_u32(smem_raw);
    const uint32_t b_res = (smem0 + 1023u) & ~1023u;
    const long long wait_limit = p.wait_cycles;
    const int ksteps = p.kchunks;
    const uint32_t b_bytes = 128u * BK * 4;                       // 128 rows (4 * tap + c) x 32 output channels
    const uint32_t ring = b_res + (uint32_t)ksteps * b_bytes;
    const uint32_t ycol_base = ring + (uint32_t)kDx3Stages * A_STAGE_BYTES;
    const int ntaps = p.KH * p.KW;
    const uint32_t bar_base = ycol_base + (uint32_t)ntaps * (kDx3Rows * 32 * 16);
    const uint32_t full_bar = bar_base;                           // [kDx3Stages]
    const uint32_t empty_bar = bar_base + 8u * kDx3Stages;        // [kDx3Stages]
    const uint32_t b_bar = bar_base + 16u * kDx3Stages;
    const uint32_t acc_full = b_bar + 8u;                         // [2] one per M tile
    const uint32_t acc_empty = acc_full + 16u;                    // [2]
    const uint32_t tmem_slot = acc_empty + 16u;
    uint32_t* tmem_slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (tmem_slot - smem0));
    const float4* ycol = reinterpret_cast<const float4*>(smem_raw + (ycol_base - smem0));
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

    if (warp == 0) {   // a lane per barrier
        if (lane < kDx3Stages) {
            mbar_init(full_bar + 8u * lane, 1);
            mbar_init(empty_bar + 8u * lane, 1);
        }
        if (lane < 2) {
            mbar_init(acc_full + 8u * lane, 1);
            mbar_init(acc_empty + 8u * lane, kDx3Epi / 32);
        }
        if (lane == 0) {
            mbar_init(b_bar, 1);
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        __syncwarp();
    }
    constexpr int tmem_cols = 256;
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_d = *tmem_slot_ptr;

    if (warp == 0) {
        // ===== producer: the weights once; per tile two M tiles (4 dy rows x 32 pixels each) x the channel chunks =====
        pdl_enter();
        if (elect_one()) {
            mbar_expect_tx(b_bar, (uint32_t)ksteps * b_bytes);
            for (int q = 0; q < ksteps; ++q) tma_load_3d(b_res + (uint32_t)q * b_bytes, &map_b, b_bar, q * BK, 0, 0);
        }
        int s = 0, it = 0;
        uint32_t phase = 0;
        bool alive = true;
        for (int tile = blockIdx.x; tile < g.tiles && alive; tile += gridDim.x) {
            int n, t;
            g.by_tiles_per_img.divmod(tile, n, t);
            const int i_base = g.R * t + g.lo;
            for (int mt = 0; mt < g.mts && alive; ++mt)
                for (int q = 0; q < ksteps; ++q, ++it) {
                    if (!mbar_wait_warp(empty_bar + 8u * s, phase ^ 1u, 0, it, wait_limit)) { alive = false; break; }
                    if (elect_one()) {
                        const uint32_t fb = full_bar + 8u * s;
                        mbar_expect_tx(fb, (uint32_t)A_STAGE_BYTES);
                        tma_load_4d(ring + (uint32_t)s * A_STAGE_BYTES, &map_a, fb, q * BK, 0, i_base + 4 * mt, n);
                    }
                    if (++s == kDx3Stages) { s = 0; phase ^= 1u; }
                }
        }
    } else if (warp == 1) {
        // ===== MMA issuer: both operands K-major =====
        const uint32_t idesc = make_idesc(0, 0, 128, BM);
        const uint64_t adesc0 = make_smem_desc(ring, 16u, 1024u, kLayoutSw128);
        const uint64_t bdesc0 = make_smem_desc(b_res, 16u, 1024u, kLayoutSw128);
        int s = 0, it = 0, n = 0;
        uint32_t phase = 0;
        bool alive = mbar_wait_warp(b_bar, 0, 1, -1, wait_limit);
        for (int tile = blockIdx.x; tile < g.tiles && alive; tile += gridDim.x, ++n) {
            for (int mt = 0; mt < g.mts && alive; ++mt) {
                // the epilogue has copied this accumulator's previous tile to shared memory (first tile: passes at once)
                if (!mbar_wait_warp(acc_empty + 8u * mt, ((uint32_t)n & 1u) ^ 1u, 1, it, wait_limit)) { alive = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int q = 0; q < ksteps; ++q, ++it) {
                    if (!mbar_wait_warp(full_bar + 8u * s, phase, 1, it, wait_limit)) { alive = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (elect_one()) {
                        const uint64_t adesc = adesc0 + (uint64_t)((uint32_t)s * (A_STAGE_BYTES >> 4));
                        const uint64_t bdesc = bdesc0 + (uint64_t)((uint32_t)q * (b_bytes >> 4));
#pragma unroll
                        for (int kk = 0; kk < BK / 8; ++kk)
                            tcgen05_mma_tf32(tmem_d + (uint32_t)(mt * 128), adesc + (uint64_t)(kk * 2), bdesc + (uint64_t)(kk * 2), idesc,
                                             (q > 0 || kk > 0) ? 1u : 0u);
                        tcgen05_commit(empty_bar + 8u * s);
                    }
                    if (++s == kDx3Stages) { s = 0; phase ^= 1u; }
                }
                if (elect_one()) tcgen05_commit(acc_full + 8u * mt);   // complete, or abandoned
            }
        }
    } else {
        // ===== epilogue: accumulators -> shared memory [tap][dy pixel][4], then gather the tile's own output pixels =====
        const int quad = warp & 3;
        const int row = quad * 32 + lane;                // dy pixel of the M tile: 32 * (row of the tile) + column
        const int slab = (warp - 2) >> 2;                // the four warps of a lane quadrant take one 32-column slab each
        const bool drains = slab * 32 < 4 * ntaps;
        pdl_enter();
        int n_it = 0;
        for (int tile = blockIdx.x; tile < g.tiles; tile += gridDim.x, ++n_it) {
            int n, t;
            g.by_tiles_per_img.divmod(tile, n, t);
            bool ok = true;
            for (int mt = 0; mt < g.mts; ++mt) {
                const bool got = mbar_wait(acc_full + 8u * mt, (uint32_t)n_it & 1u, 2, n_it, wait_limit);
                ok = __all_sync(0xffffffffu, got) && ok;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                uint32_t r[32];
                if (drains) tmem_ld_32x32b_x32(tmem_d + ((uint32_t)(quad * 32) << 16) + (uint32_t)(mt * 128 + slab * 32), r);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                // in registers: back to the MMA warp with it before anything is stored
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acc_empty + 8u * mt) : "memory");
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int tap = slab * 8 + q;
                    if (tap < ntaps) {
                        const uint32_t addr = ycol_base + (uint32_t)(((tap * kDx3Rows * 32) + mt * 128 + row) * 16);
                        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(__uint_as_float(r[4 * q])),
                                     "f"(__uint_as_float(r[4 * q + 1])), "f"(__uint_as_float(r[4 * q + 2])),
                                     "f"(__uint_as_float(r[4 * q + 3])) : "memory");
                    }
                }
            }
            asm volatile("bar.sync 1, %0;" ::"n"(kDx3Epi) : "memory");
            if constexpr (KH_ > 0) dx3_gather_pairs<KH_, KW_>(p, g, ycol, n, t, ok, warp - 2, lane);
            else dx3_gather(p, g, ycol, n, t, ok, (int)threadIdx.x - 64);
            asm volatile("bar.sync 1, %0;" ::"n"(kDx3Epi) : "memory");   // the products are consumed: the next tile may overwrite them
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"(tmem_cols) : "memory");
    }
}

}  // namespace
}  // namespace dcg

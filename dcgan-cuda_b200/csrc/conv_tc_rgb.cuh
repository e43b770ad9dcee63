// conv_fwd_rgb_kernel: forward of a layer with <= 4 input channels, straight from its image.  Included by conv_tc.cu only.
#pragma once

namespace dcg {
namespace {

// ---- forward of a <= 4-channel layer: tile operands built in the CTA -----------------------------------
// A 3-channel pixel is 12 bytes, which TMA cannot step by.  Through a zero-bordered 4-channel copy of the image it can fetch
// the 32-float window of a kernel row per output pixel, but that is a launch more, twice the reduction steps, and 128-byte
// rows at 32-byte steps come in at 16 bytes per clock.  Here eight warps copy the patch of the image under a tile to shared
// memory (one TMA load where the image's rows are TMA rows, else cp.async; zeros beyond the border) and build the im2col rows from it, in the swizzled K-major layout of the tensor
// core: 16 (or 32) places per kernel row, of which KW * C are used; the weights come in the same order from where they are.
// Persistent, one CTA per SM: the patches of the next tiles are copied, and the next rows built, while this tile's products and
// its epilogue run (two operand tiles, two accumulators).
// An operand tile holds all kernel rows, which limits the layers: rows of up to 16 values (KW * C) up to 5 x 5 with three channels or
// 4 x 4 with four (with a stride and 96 or 128 outputs 5 x 5 x 3 only over small images), rows of more than 16 values only up to four of
// them.  The others - 5 x 5 x 4, 6 x 6 x 3, 7 x 7 x 3 - keep the two launches.
// What bounds it is the shared-memory pipe: a tile of 5 x 5 x 3 -> 64 is 800 clocks of building (8-byte reads of a lane, which a
// lane stride of an even number of floats spreads over all banks, and one 16-byte store per four places) and 256 clocks to
// stage the output, which TMA stores.  (Rows without places between them, element by element through a table: 2300 clocks; the
// patch in 4-byte copies: 500 to 1700; the output turned in shared memory to be stored by the threads: 2900.)
// 3 -> 64 channels, 5 x 5 / stride 2, of 8 / 64 / 128 / 256 images of 64 x 64: 6.1 / 9.5 / 13.8 / 23.2 us; through the 4-channel
// copy, two launches, 10.2 / 15.0 / 22.4 / 38.7.
struct RgbArgs {
    int kwc;           // KW * C, used places of a kernel row
    int chunks;        // of 32 along k
    int ksteps;        // MMAs of 8 along k
    int rows, row_len; // the patch: rows of all its images, floats per row
    int pitch;         // floats from one row of the patch to the next, even
    int tma;           // patches come by TMA: they begin on 16 bytes, up to three floats before the first pixel
    unsigned patch_tx; // bytes of such a load
    int patch_bytes, patches;   // 2 to 4 of them: a copy takes about as long as two tiles
    int tiles;
};
constexpr int kRgbBuilders = 256, kRgbEpi = 256, kRgbThreads = kRgbBuilders + kRgbEpi + 32;
constexpr int kRgbMaxChunks = 8;
constexpr int kRgbStage = 32 * 128;   // bytes of 32 output pixels x 32 channels; two of them per epilogue warp

// Shared memory behind the 1 KB of alignment slack: operand tiles [2], weights, staged output, patches, barriers.
__host__ __device__ constexpr size_t rgb_smem(int chunks, int bn, size_t patch_bytes)
{
    return 1024 + (size_t)chunks * (2 * A_STAGE_BYTES + bn * BK * 4) + kRgbEpi / 32 * 2 * kRgbStage + patch_bytes + 192;
}

__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2, int c3)
{
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
                 ::"l"(map), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

// PLACES of a kernel row; EVEN: pixels of a tile row are an even number of floats apart.
template <int PLACES, bool EVEN>
__global__ void __launch_bounds__(kRgbThreads, 1)
conv_fwd_rgb_kernel(const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_out, const __grid_constant__ CUtensorMap map_raw,
                    const __grid_constant__ CUtensorMap map_pre, const __grid_constant__ CUtensorMap map_gate, const __grid_constant__ CUtensorMap map_x,
                    const __grid_constant__ Params p,
                    const __grid_constant__ RgbArgs g, const float* __restrict__ x)
{
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem0 = smem_u32(smem_raw);
    const uint32_t a_base = (smem0 + 1023u) & ~1023u;
    const uint32_t a_bytes = (uint32_t)g.chunks * A_STAGE_BYTES, b_chunk = (uint32_t)p.bn * BK * 4;
    const uint32_t b_base = a_base + 2u * a_bytes;
    const uint32_t stage_base = b_base + (uint32_t)g.chunks * b_chunk;
    const uint32_t patch_base = stage_base + (uint32_t)(kRgbEpi / 32 * 2 * kRgbStage);   // each patch on 128 bytes
    const uint32_t bar_base = (patch_base + (uint32_t)(g.patches * g.patch_bytes) + 7u) & ~7u;
    const uint32_t a_full = bar_base, a_empty = bar_base + 16u;              // [2] operand tile built / read by its MMAs
    const uint32_t acc_full = bar_base + 32u, acc_empty = bar_base + 48u;    // [2] accumulator complete / drained
    const uint32_t gate_bar = bar_base + 64u;                                // [8] an epilogue warp's gate values have landed
    const uint32_t patch_bar = bar_base + 128u;                              // [4] a patch has landed
    const uint32_t b_bar = bar_base + 160u, tmem_slot = bar_base + 168u;
    const long long wait_limit = p.wait_cycles;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    constexpr int kMmaWarp = (kRgbBuilders + kRgbEpi) / 32;
    auto generic = [&](uint32_t at) { return smem_raw + (at - smem0); };

    int tmem_cols = 32;
    while (tmem_cols < 2 * p.bn) tmem_cols <<= 1;
    if (warp == kMmaWarp) {
        if (lane < 2) {
            mbar_init(a_full + 8u * lane, kRgbBuilders / 32);
            mbar_init(a_empty + 8u * lane, 1);
            mbar_init(acc_full + 8u * lane, 1);
            mbar_init(acc_empty + 8u * lane, kRgbEpi / 32);
        }
        if (lane < kRgbEpi / 32) mbar_init(gate_bar + 8u * lane, 1);
        if (lane < 4) mbar_init(patch_bar + 8u * lane, 1);
        if (lane == 0) {
            mbar_init(b_bar, 1);
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_out) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_d = *reinterpret_cast<uint32_t*>(generic(tmem_slot));

    auto origin = [&](int tile, int& j0, int& i0, int& n0) {
        p.by_tiles_w.divmod(tile, n0, j0);
        p.by_tiles_h.divmod(n0, n0, i0);
        j0 *= p.TW; i0 *= p.TH; n0 *= p.TN;
    };

    if (warp < kRgbBuilders / 32) {
        // ===== builders =====
        const int rows_per_img = (p.TH - 1) * p.sh + p.KH, line = p.W * p.C;
        bool alive = true;   // (a warp that gave up loads nothing more: nobody would wait for it before the CTA leaves)
        auto copy = [&](int tile, int buf) {   // by TMA, or a warp per row of the patch; a group even where there is no such tile, for groups are counted
            int j0, i0, n0;
            origin(tile, j0, i0, n0);
            const int first = (j0 * p.sw - p.pl) * p.C;
            if (g.tma) {
                if (warp == 0 && alive && tile < g.tiles && elect_one()) {
                    mbar_expect_tx(patch_bar + 8u * buf, g.patch_tx);
                    tma_load_3d(patch_base + (uint32_t)(buf * g.patch_bytes), &map_x, patch_bar + 8u * buf, first & ~3, i0 * p.sh - p.pt, n0);
                }
                return;
            }
            int img = 0, r = warp;
            for (int row = warp; row < (tile < g.tiles ? g.rows : 0); row += kRgbBuilders / 32) {
                while (r >= rows_per_img) { r -= rows_per_img; ++img; }
                const int h = i0 * p.sh - p.pt + r, n = n0 + img;
                const bool in_row = h >= 0 && h < p.H && n < p.N;
                const float* src = x + ((size_t)(in_row ? n : 0) * p.H + (in_row ? h : 0)) * (size_t)line;
                const uint32_t dst = patch_base + (uint32_t)(buf * g.patch_bytes) + (uint32_t)(row * g.pitch) * 4u;
                for (int e = lane; e < g.row_len; e += 32) {
                    const bool in = in_row && first + e >= 0 && first + e < line;
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + 4u * e), "l"(src + (in ? first + e : 0)), "r"(in ? 4 : 0) : "memory");
                }
                r += kRgbBuilders / 32;
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        const int pixel = threadIdx.x & (BM - 1), part = threadIdx.x >> 7;
        const int tw = pixel % p.TW, th = (pixel / p.TW) % p.TH, tn = pixel / (p.TW * p.TH);
        const int at = (tn * rows_per_img + th * p.sh) * g.pitch + tw * p.sw * p.C;
        pdl_enter();
        const int step = gridDim.x;
        int ahead = blockIdx.x;   // the next tile to copy, and where to
        for (int b = 0; b < g.patches - 1; ++b, ahead += step) copy(ahead, b);
        int buf_in = g.patches - 1, buf_out = 0;
        uint32_t phase_out = 0;
        int n = 0;
        for (int tile = blockIdx.x; tile < g.tiles; tile += gridDim.x, ++n) {
            const int buf = n & 1;
            if (g.tma) alive = alive && mbar_wait_warp(patch_bar + 8u * buf_out, phase_out, 4, n, wait_limit);
            else if (g.patches == 4) asm volatile("cp.async.wait_group 2;" ::: "memory");
            else if (g.patches == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
            else asm volatile("cp.async.wait_group 0;" ::: "memory");
            asm volatile("bar.sync 1, %0;" ::"n"(kRgbBuilders) : "memory");   // the patch is there, and nobody reads that of the tile before any more
            copy(ahead, buf_in);
            ahead += step;
            if (++buf_in == g.patches) buf_in = 0;
            const uint32_t patch = patch_base + (uint32_t)(buf_out * g.patch_bytes);
            if (++buf_out == g.patches) { buf_out = 0; phase_out ^= 1u; }
            int j0, i0, n0;
            origin(tile, j0, i0, n0);
            const int shift = g.tma ? (j0 * p.sw - p.pl) * p.C & 3 : 0;   // of the first pixel in its row
            // (a warp that gave up goes on to the barriers of the others)
            if (alive) alive = mbar_wait_warp(a_empty + 8u * buf, ((uint32_t)(n >> 1) & 1u) ^ 1u, 0, n, wait_limit);
            if (!alive) continue;
            const bool odd = EVEN && (shift & 1) != 0;
            const float* src = reinterpret_cast<const float*>(generic(patch)) + at + (odd ? shift - 1 : shift);
            uint8_t* dst = generic(a_base + (uint32_t)buf * a_bytes) + pixel * 128;
#pragma unroll 5
            for (int di = 0; di < p.KH; ++di, src += g.pitch) {
#pragma unroll
                for (int i = 0; i < PLACES / 8; ++i) {   // the threads of a pixel take four places in turn
                    const int q = 4 * (part + 2 * i), u = di * (PLACES / 4) + part + 2 * i;
                    float4 v;
                    if constexpr (EVEN) {   // three reads at an even place, whether the first value lies there or one further on
                        const float2 a = *reinterpret_cast<const float2*>(src + q), b = *reinterpret_cast<const float2*>(src + q + 2),
                                     c = *reinterpret_cast<const float2*>(src + q + 4);
                        v = odd ? make_float4(a.y, b.x, b.y, c.x) : make_float4(a.x, a.y, b.x, b.y);
                    } else {
                        v = make_float4(src[q], src[q + 1], src[q + 2], src[q + 3]);
                    }
                    // the places beyond the row's last hold another pixel's values
                    v.x = q < g.kwc ? v.x : 0.f; v.y = q + 1 < g.kwc ? v.y : 0.f;
                    v.z = q + 2 < g.kwc ? v.z : 0.f; v.w = q + 3 < g.kwc ? v.w : 0.f;
                    *reinterpret_cast<float4*>(dst + (u >> 3) * A_STAGE_BYTES + (((u & 7) ^ (pixel & 7)) << 4)) = v;
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic-proxy writes -> tensor core reads
            __syncwarp();
            if (lane == 0 && n != p.skip_stage) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(a_full + 8u * buf) : "memory");
        }
    } else if (warp == kMmaWarp) {
        // ===== the weights, then the products: A K-major, B MN-major (chunks of 32 columns 4096 B apart, 4-row groups 512 B apart) =====
        pdl_enter();
        if (elect_one()) {
            mbar_expect_tx(b_bar, (uint32_t)g.chunks * b_chunk);
            for (int q = 0; q < g.chunks; ++q) tma_load_4d(b_base + (uint32_t)q * b_chunk, &map_b, b_bar, 0, 0, q * (BK / PLACES), 0);
        }
        const uint32_t idesc = make_idesc(0, 1, p.bn, BM);
        const uint64_t adesc0 = make_smem_desc(a_base, 16u, 1024u, kLayoutSw128);
        const uint64_t bdesc0 = make_smem_desc(b_base, 4096u, 512u, kLayoutSw128Base32);
        bool alive = mbar_wait_warp(b_bar, 0, 1, -1, wait_limit);
        int n = 0;
        for (int tile = blockIdx.x; tile < g.tiles && alive; tile += gridDim.x, ++n) {
            const int buf = n & 1;
            const uint32_t phase = (uint32_t)(n >> 1) & 1u;
            alive = mbar_wait_warp(acc_empty + 8u * buf, phase ^ 1u, 1, n, wait_limit) && mbar_wait_warp(a_full + 8u * buf, phase, 1, n, wait_limit);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one()) {
                if (alive) {
                    const uint64_t adesc = adesc0 + (uint64_t)((uint32_t)buf * (a_bytes >> 4));
                    for (int k = 0; k < g.ksteps; ++k)
                        tcgen05_mma_tf32(tmem_d + (uint32_t)(buf * p.bn), adesc + (uint64_t)((k >> 2) * (A_STAGE_BYTES >> 4) + (k & 3) * 2),
                                         bdesc0 + (uint64_t)((uint32_t)(k >> 2) * (b_chunk >> 4) + (uint32_t)(k & 3) * 64u), idesc, k > 0 ? 1u : 0u);
                    tcgen05_commit(a_empty + 8u * buf);
                }
                tcgen05_commit(acc_full + 8u * buf);   // complete, or abandoned
            }
        }
    } else {
        // ===== epilogue: thread = accumulator row; the two warps of a lane quadrant take alternate 32-column slabs; each result of the
        // chain goes through the warp's staging buffers (rows of 128 bytes, swizzled) and out as one TMA store =====
        const int w = warp - kRgbBuilders / 32, quad = warp & 3, first = w >> 2, nslabs = p.bn >> 5;
        const int r0 = quad * 32, tw = r0 % p.TW, th = (r0 / p.TW) % p.TH, tn = r0 / (p.TW * p.TH);   // the warp's first pixel
        const EpilogueArgs& e = p.ep;
        const uint32_t stage = stage_base + (uint32_t)(w * 2 * kRgbStage);
        uint32_t turn = 0;   // without a gate the two buffers take turns, else the second one holds its values
        pdl_enter();
        int n = 0;
        uint32_t gates = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < g.tiles; tile += gridDim.x, ++n) {
            const int buf = n & 1;
            int j, i, img;
            origin(tile, j, i, img);
            j += tw; i += th; img += tn;
            auto load_gate = [&](int sl) {
                __syncwarp();
                if (lane == 0) {
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // (the values before them have been read)
                    mbar_expect_tx(gate_bar + 8u * w, kRgbStage);
                    tma_load_4d(stage + kRgbStage, &map_gate, gate_bar + 8u * w, sl * 32, j, i, img);
                }
            };
            if (ok && e.gate && first < nslabs) load_gate(first);
            ok = ok && mbar_wait_warp(acc_full + 8u * buf, (uint32_t)(n >> 1) & 1u, 2, n, wait_limit);   // (waits in vain once at most)
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int sl = first; sl < nslabs; sl += 2) {
                const int c0 = sl * 32;
                float v[32];
                {
                    uint32_t r[32];
                    tmem_ld_32x32b_x32(tmem_d + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * p.bn + c0), r);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int q = 0; q < 32; ++q) v[q] = __uint_as_float(r[q]);
                }
                if (sl + 2 >= nslabs) {   // this warp's last read of the buffer: hand it back to the MMA warp
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acc_empty + 8u * buf) : "memory");
                }
                auto put = [&](const CUtensorMap* map) {
                    const uint32_t at = stage + turn;
                    if (!e.gate) turn ^= kRgbStage;
                    if (lane == 0) {   // the store that read this buffer has done so
                        if (e.gate) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                        else asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                    }
                    __syncwarp();
                    uint8_t* to = generic(at) + lane * 128;
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        *reinterpret_cast<float4*>(to + ((q ^ (lane & 7)) << 4)) = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (ok && lane == 0) tma_store_4d(map, at, c0, j, i, img);
                };
                if (e.raw_out) put(&map_raw);
                if (e.bias) {
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const float4 b = __ldg(reinterpret_cast<const float4*>(e.bias + c0) + q);
                        v[4 * q] = __fadd_rn(v[4 * q], b.x); v[4 * q + 1] = __fadd_rn(v[4 * q + 1], b.y);
                        v[4 * q + 2] = __fadd_rn(v[4 * q + 2], b.z); v[4 * q + 3] = __fadd_rn(v[4 * q + 3], b.w);
                    }
                }
                if (e.pre_act) put(&map_pre);
                act_apply_all(v, e.act, e.alpha);
                if (e.gate) {
                    ok = ok && mbar_wait_warp(gate_bar + 8u * w, gates & 1u, 3, n, wait_limit);
                    ++gates;
                    const uint8_t* from = generic(stage + kRgbStage) + lane * 128;
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const float4 gq = *reinterpret_cast<const float4*>(from + ((q ^ (lane & 7)) << 4));
                        float four[4] = {v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]};
                        const float gate[4] = {gq.x, gq.y, gq.z, gq.w};
                        act_grad_apply_all(four, gate, e.gate_act, e.gate_alpha);
                        v[4 * q] = four[0]; v[4 * q + 1] = four[1]; v[4 * q + 2] = four[2]; v[4 * q + 3] = four[3];
                    }
                    if (ok && sl + 2 < nslabs) load_gate(sl + 2);
                }
                put(&map_out);
            }
            if (nslabs <= first) {   // a warp without a slab still has to hand the buffer back
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acc_empty + 8u * buf) : "memory");
            }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"(tmem_cols) : "memory");
    }
}

}  // namespace
}  // namespace dcg

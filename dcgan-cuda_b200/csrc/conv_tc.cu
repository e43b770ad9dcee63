// tcgen05 implicit-GEMM convolution kernels (TF32 operands, fp32 accumulation in TMEM).
//
// One kernel template covers the three operators; each is a GEMM D[M x N] += A[M x K] B[K x N]
// whose operand tiles are fetched straight from the NHWC / HWIO tensors by TMA - no im2col
// buffer, no zero-inserted gradient, no weight repacking ever exists in memory:
//
//   FWD  y[pix, o]      = sum_{tap, c} x[pix*s + tap - pad, c] * k[tap, c, o]
//        A: x through a 4-D tiled map with traversal stride s, box (32 c, TW, TH, TN) -> 128 output
//           pixels x 32 channels, K-major; taps that fall outside x are zero-filled by TMA, which is
//           the reference's "skip out-of-range taps" (src/cpu/ops.hxx:236-243).
//        B: k as [tap][c][o], o contiguous -> MN-major tile (32 c x BN o).
//   DX   dx[pix, c]     = sum_{tap, o} dy[(pix + pad - tap)/s, o] * k[tap, c, o]
//        split by output parity class (pix mod s): inside a class the taps with matching parity
//        read a dense, stride-1 window of dy, so none of the 4x multiplications by inserted zeros
//        of the reference's formulation (src/gpu/conv2d_gemm.hh:396-412) is ever issued.
//        A: dy, box (32 o, TW, TH, TN), K-major.  B: k rows c, 32 o contiguous, K-major.
//   DK   dk[tap, c, o]  = sum_{pix} x[pix*s + tap - pad, c] * dy[pix, o]
//        reduction over pixels; both operands have the reduction index outermost in memory, so
//        both tiles are MN-major (32 pixels x 128 channels / BN channels), 5-D maps.
//
// CTA = 320 threads: warp 0 issues TMA, warp 1 owns TMEM and issues tcgen05.mma (both walked by the
// whole warp with one elected lane issuing), warps 2-9 - two per TMEM lane quadrant - drain the
// accumulator (tcgen05.ld) through the fused epilogue (raw / bias / pre-activation / activation /
// activation-gradient gate) into HBM; in the 3xTF32 variant they also build the residual tiles of
// every stage.  A ring of smem stages (A 16 KB + B BN*128 B, 128-byte swizzle; 7 deep with one
// CTA per SM) is handed over with mbarriers: TMA complete_tx -> MMA, tcgen05.commit -> TMA.
// The K partitions of one tile form a thread-block cluster: each writes the other partitions' shares of its
// fp32 partial tile to scratch (L2-resident), the cluster meets at a hardware barrier, and every CTA then
// adds the others' partials to its own share, in partition order (deterministic), and finishes it, fused
// epilogue included - one launch per convolution.  Kernel gradients of few tiles take more partitions than a
// cluster holds and a second launch that adds them (dk_finish_kernel).
//
// Every wait is bounded: a barrier that does not complete within ~1 s makes the waiting role
// record an error code in a device status word and leave; TMEM is always released.
//
// This file is the host side (tensor maps, planning, the plan cache, launches, entry points); the
// device code of this translation unit sits in the headers it includes:
//   conv_tc_common.cuh   constants, kernel parameters, PTX wrappers, descriptors
//   conv_tc_kernel.cuh   conv_tc_kernel<MODE, KIND>, the general kernel described above
//   conv_tc_dxf.cuh      conv_dxf_kernel: input gradient with all parity classes of a pixel tile in one
//                        CTA, their accumulators merged into wide MMAs
//   conv_tc_walk.cuh     conv_tc_walk_kernel: forward and input gradient of layers with more tiles than SMs
//   conv_tc_short.cuh    conv_fwd_short_kernel: the short-K forward GEMMs of the 3-channel layers as
//                        persistent CTAs with resident weights and a double-buffered accumulator
//   conv_tc_rgb.cuh      conv_fwd_rgb_kernel: forward of a <= 4-channel layer straight from its image
//   conv_tc_dx3.cuh      conv_dx3_kernel: input gradient of a 3-channel layer, GEMM + gather in one kernel
//   conv_tc_narrow.cuh   repack, partition-finish and gather helpers of the 3-channel layers
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "common.cuh"
#include "conv.cuh"

#include "conv_tc_common.cuh"
#include "conv_tc_kernel.cuh"
#include "conv_tc_dxf.cuh"
#include "conv_tc_walk.cuh"
#include "conv_tc_short.cuh"
#include "conv_tc_rgb.cuh"
#include "conv_tc_dx3.cuh"
#include "conv_tc_narrow.cuh"

namespace dcg {
namespace {

// ---- host side: tensor maps ---------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn()
{
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(sym);
    });
    return fn;
}

std::atomic<unsigned long long> g_maps_encoded{0};

// dims/strides innermost first; strides[i] is the byte stride of dimension i+1.
int encode_map(CUtensorMap* map, const void* base, int rank, const cuuint64_t* dims, CUtensorMapSwizzle swizzle,
               const cuuint64_t* strides, const cuuint32_t* box, const cuuint32_t* estrides)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fail(DCG_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    g_maps_encoded.fetch_add(1, std::memory_order_relaxed);
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, (cuuint32_t)rank, const_cast<void*>(base), dims,
                          strides, box, estrides, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        return fail(DCG_ERR_CUDA,
                    "cuTensorMapEncodeTiled failed (%d): rank %d dims [%llu,%llu,%llu,%llu,%llu] box [%u,%u,%u,%u,%u]",
                    (int)r, rank, (unsigned long long)dims[0], (unsigned long long)dims[1],
                    (unsigned long long)(rank > 2 ? dims[2] : 0), (unsigned long long)(rank > 3 ? dims[3] : 0),
                    (unsigned long long)(rank > 4 ? dims[4] : 0), box[0], box[1], rank > 2 ? box[2] : 0,
                    rank > 3 ? box[3] : 0, rank > 4 ? box[4] : 0);
    }
    return DCG_OK;
}

int encode_map(CUtensorMap* map, const void* base, int rank, const cuuint64_t* dims, bool mn_major,
               const cuuint64_t* strides, const cuuint32_t* box, const cuuint32_t* estrides)
{
    return encode_map(map, base, rank, dims, mn_major ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B, strides, box, estrides);
}

// Activation [N, Hh, Ww, Cc] as a 4-D map (c, w, h, n) with a (32, tw, th, tn)-element box and
// traversal strides (1, sw, sh, 1).
int map_act_4d(CUtensorMap* map, const float* base, int N, int Hh, int Ww, int Cc, int tw, int th, int tn,
               int sw, int sh, bool mn_major = false)
{
    const cuuint64_t dims[4] = {(cuuint64_t)Cc, (cuuint64_t)Ww, (cuuint64_t)Hh, (cuuint64_t)N};
    const cuuint64_t strides[3] = {(cuuint64_t)Cc * 4, (cuuint64_t)Ww * Cc * 4, (cuuint64_t)Hh * Ww * Cc * 4};
    const cuuint32_t box[4] = {32, (cuuint32_t)(tw * sw), (cuuint32_t)(th * sh), (cuuint32_t)tn};
    const cuuint32_t es[4] = {1, (cuuint32_t)sw, (cuuint32_t)sh, 1};
    return encode_map(map, base, 4, dims, mn_major, strides, box, es);
}

// Activation [N, Hh, Ww, Cc] as a 5-D map (c%32, w, h, n, c/32): box (32, tw, th, tn, chunks) lands in
// shared memory as [chunk][pixel][32 channels], the MN-major operand layout.
int map_act_5d(CUtensorMap* map, const float* base, int N, int Hh, int Ww, int Cc, int tw, int th, int tn,
               int sw, int sh, int chunks)
{
    const cuuint64_t dims[5] = {32, (cuuint64_t)Ww, (cuuint64_t)Hh, (cuuint64_t)N, (cuuint64_t)(Cc / 32)};
    const cuuint64_t strides[4] = {(cuuint64_t)Cc * 4, (cuuint64_t)Ww * Cc * 4, (cuuint64_t)Hh * Ww * Cc * 4, 128};
    const cuuint32_t box[5] = {32, (cuuint32_t)(tw * sw), (cuuint32_t)(th * sh), (cuuint32_t)tn, (cuuint32_t)chunks};
    const cuuint32_t es[5] = {1, (cuuint32_t)sw, (cuuint32_t)sh, 1, 1};
    return encode_map(map, base, 5, dims, true, strides, box, es);
}

int pow2_ceil(int v)
{
    int r = 1;
    while (r < v) r <<= 1;
    return r;
}

// 128 (or `total`) pixels as a (tw, th, tn) box: w first, then h, then images.
void pixel_tile(int total, int Wd, int Hd, int& tw, int& th, int& tn)
{
    tw = pow2_ceil(Wd); if (tw > total) tw = total;
    th = pow2_ceil(Hd); if (th > total / tw) th = total / tw;
    tn = total / (tw * th);
}

// The same, or the box that covers the image with the fewest copies where that is fewer: 17 x 7 of the 128 rows for images
// of 51 x 75 (429 boxes of 13 images; 64 x 2 takes 494).  `whole`: every row of the tile has to hold a pixel.
void pixel_tile_fit(int total, int Wd, int Hd, int Nd, int sw, int sh, bool whole, int& tw, int& th, int& tn)
{
    pixel_tile(total, Wd, Hd, tw, th, tn);
    auto boxes = [&](int a, int b, int c) { return (long long)((Wd + a - 1) / a) * ((Hd + b - 1) / b) * ((Nd + c - 1) / c); };
    long long best = boxes(tw, th, tn);
    // fewer images than fit: nothing is loaded for the others (one sampled image 41.3 -> 36.2 us)
    if (!whole && tn > Nd) tn = Nd;
    for (int a = 1; a <= total && a * sw <= 256; whole ? a *= 2 : ++a)
        for (int b = 1; a * b <= total && b * sh <= 256; whole ? b *= 2 : ++b) {
            int c = total / (a * b);
            if (!whole && c > Nd) c = Nd;
            if (boxes(a, b, c) < best) { best = boxes(a, b, c); tw = a; th = b; tn = c; }
        }
}

struct Plan {
    Params p;
    int grid;
    size_t smem;
    // scratch layout: [partial tiles of the K partitions][padded 4-channel input xp][repacked weights
    // k4], each part 256-byte aligned; the last two only exist for narrow-channel layers
    size_t partial_bytes = 0, xp_bytes = 0, k4_bytes = 0, ws_bytes = 0;
    int Hp = 0, Wp = 0;   // padded input extent of a narrow-channel layer
    // DX of a narrow-channel layer (GEMM + gather): p describes the 1x1 FWD problem; the transposed
    // weights k2 and the GEMM result ycol follow the partial tiles in the scratch area
    int Jp = 0;
    size_t k2_bytes = 0, ycol_bytes = 0;
    size_t k2_off() const { return align_up(partial_bytes, 256); }
    size_t ycol_off() const { return k2_off() + align_up(k2_bytes, 256); }
    size_t xp_off() const { return align_up(partial_bytes, 256); }
    size_t k4_off() const { return xp_off() + align_up(xp_bytes, 256); }
};

// DCG_TC_SPLITS / DCG_TC_STAGES (environment, read once) pin the K partitioning and the pipeline
// depth for experiments; unset or 0 leaves the heuristics below in charge.
int env_int(const char* name)
{
    const char* v = getenv(name);
    return v ? atoi(v) : 0;
}

// Set by the entry points for the duration of a call: plan for the 3xTF32 variant.
thread_local int t_plan_x3 = 0;
struct PlanX3 {
    int saved;
    explicit PlanX3(bool x3) : saved(t_plan_x3) { t_plan_x3 = x3 ? 1 : 0; }
    ~PlanX3() { t_plan_x3 = saved; }
};

// How many clusters of s CTAs with one CTA's full shared memory each are resident at a time.
int cluster_fit(int s)
{
    constexpr int kDevices = 64;
    static std::mutex mutex;
    static int fit[kDevices][kMaxCluster + 1];   // 0: not asked yet
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) { cudaGetLastError(); return sm_count() / s; }
    std::lock_guard<std::mutex> lock(mutex);
    int& f = fit[dev][s];
    if (f == 0) {
        auto kernel = conv_tc_kernel<MODE_FWD, kShared>;
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)(s * sm_count()));
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = kMaxSmem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)s; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) { cudaGetLastError(); n = sm_count() / s; }
        f = n > 0 ? n : -1;
    }
    return f;
}

// K partitions of a tile.  Measured on every DCGAN layer at batch 64 (per-CTA timelines, partition
// counts 1..8 forced): the shortest launch is the one with about ONE CTA per SM - a deeper pipeline
// per CTA and half the partial-tile traffic beat a second resident CTA (e.g. the 256 -> 512 forward
// layer: 18.5 us with 4 partitions = 128 CTAs against 22.3 us with 8 = 256; the 64 -> 128 kernel gradient with
// the channel roles swapped: 25.0 us with 25 taps x 5 = 125 CTAs against 27.0 us with 25 x 8 = 200, 39.8 us
// against 46.7 us over 128 images).
int choose_splits(int tiles, int min_stages_per_tile, int ctas_per_sm = 1)
{
    static const int forced = env_int("DCG_TC_SPLITS");
    if (forced > 0) {
        int f = forced <= min_stages_per_tile ? forced : (min_stages_per_tile > 0 ? min_stages_per_tile : 1);
        return f > kMaxCluster ? kMaxCluster : f;
    }
    const int sms = sm_count();
    if (tiles >= sms) return 1;
    int s = (ctas_per_sm * sms) / tiles;
    const int cap = min_stages_per_tile / 4;         // keep at least 4 K stages per CTA
    if (s > cap) s = cap;
    if (s > kMaxCluster) s = kMaxCluster;   // (9 to 16, the non-portable sizes, were measured: no launch got shorter)
    // A cluster lives inside one GPC, so fewer clusters are resident than the SM count suggests (15 of 8 CTAs on the
    // 148-SM part, not 18), and one cluster too many is a second wave: the 64 -> 128 forward of 8 images took 16.7 us as
    // 16 clusters of 8 and takes 10.4 us as 16 of 6.
    while (s > 1 && tiles > cluster_fit(s)) --s;
    return s < 1 ? 1 : s;
}

// Shared memory of one of two CTAs per SM holds three stages up to this accumulator width.
constexpr int kMaxSharedWidth = 160;

// Accumulator width (columns of one tile) and K partitions for n_ch output columns: the quickest of the widths that split
// n_ch evenly, by a model of the launch in SM clocks.  Its terms were read off per-CTA timelines:
//   * a stage (K = 32) takes 300 clocks up to 128 columns - four MMAs of 69, the rest the hand-over, which kDual hides - and
//     up to 512 at 256, where the MMAs alone set the pace (the full rate of the tensor core); the first is 1200 clocks away;
//   * 3xTF32 takes 1150 clocks at 64 columns and 1550 at 128, the larger part of them to take the A operand apart;
//   * the epilogue takes time per column, and two to three times that where partial tiles go through L2;
//   * up to kMaxSharedWidth columns two CTAs share an SM, so that one's epilogue hides behind the other's stages.
// 256 columns win where the tiles still fill the chip: the 128 -> 256 forward of 256 images takes 40.4 us for 46.7 with 128,
// the 256 -> 512 kernel gradient 46 for 53.  They lose where they need more partitions (256 -> 512 forward of 64 images: 22
// for 17), and where partitions would be many, narrow tiles win (128 -> 256 forward of 8 images, 64 columns: 8.8 for 10.1).
// Channel counts between the powers of two get one tile instead of two (96 -> 160 forward of 13 images of 51 x 75: 35 for 59).
// `m_count`: tiles along the other axis, times classes or taps; `store_cost`: clocks per column of an unpartitioned epilogue;
// `loads`: TMA loads per stage, of which two are in the figures above; `b_pieces`: B comes in loads of 32 columns.
// `partials_bytes` (kernel gradients): partial tiles that a second launch adds may take so much scratch.  A tile then has as many
// partitions as fill the SMs, not the eight CTAs of a cluster: the launch costs about 4 us, which long reductions over few tiles
// earn many times over (1 x 1, 8 -> 16 channels, 20 images of 64 x 64: 46 us in one cluster of eight, 10.4 in 148 partitions;
// 3 x 3, 96 -> 160, 13 images of 75 x 51: 49 and 30; 64 -> 128 of 64 images, 3xTF32: 53 and 42).  Its price in the model, 6500 clocks and
// one per 2500 bytes, leaves the line where it pays: of ninety layers drawn at random (1 x 1 to 5 x 5, 8 to 256 channels, up to 40 GFLOP)
// it is chosen for 22 in TF32, nineteen of them 7 % to 2.7 times quicker than the cluster and three 1, 3 and 10 % slower (1 x 1,
// 32 -> 128, 39 images of 8 x 38: 8.7 and 9.7), and for 45 in 3xTF32, all of them 1.1 to 6.9 times quicker.  Of the 42 that keep the
// cluster in TF32 half are quicker so (down to 0.77); eleven would gain 8 to 26 %.
struct Tiling {
    int bn, n_tiles, splits, grid;
    bool second_launch, walk;
    double cost;
};
Tiling choose_tiling(int m_count, int n_ch, int granule, int min_stages, int max_stages, int store_cost, int loads = 2, bool b_pieces = false,
                     size_t partials_bytes = 0, bool may_walk = false)
{
    static const int no_walk = env_int("DCG_TC_NO_WALK");
    if (no_walk || t_plan_x3) may_walk = false;
    static const int forced = env_int("DCG_TC_BN");
    const int sms = sm_count();
    const int widest = t_plan_x3 ? 128 : 256;   // 3xTF32: accumulators, residuals and A operands share TMEM
    Tiling best{};
    for (int n_tiles = (n_ch + widest - 1) / widest; n_tiles <= (n_ch + 63) / 64; ++n_tiles) {
        Tiling t;
        t.bn = ((n_ch + n_tiles - 1) / n_tiles + granule - 1) / granule * granule;
        if (forced >= granule && forced <= widest && n_ch >= forced) t.bn = forced / granule * granule;
        t.n_tiles = (n_ch + t.bn - 1) / t.bn;
        t.splits = choose_splits(m_count * t.n_tiles, min_stages);
        t.grid = m_count * t.n_tiles * t.splits;
        const int waves = (t.grid + sms - 1) / sms;
        const double stage = t_plan_x3 ? 750.0 + 6.25 * t.bn
                             : t.bn > 128 ? 300.0 + (t.bn - 128) * (212.0 / 128) : t.bn <= 64 && waves == 1 ? 250.0 : 300.0;
        const double loop = 1200.0 + (max_stages + t.splits - 1) / t.splits * (stage + 20.0 * (loads - 2 + (b_pieces ? (t.bn + 31) / 32 - 1 : 0)));
        const double epilogue = t.bn * (t.splits > 1 ? 55.0 : (double)store_cost);
        t.cost = t.bn <= kMaxSharedWidth && !t_plan_x3 ? waves * loop + epilogue : waves * (loop + epilogue);
        t.second_launch = false;
        t.walk = may_walk && t.splits == 1 && t.grid > sms;
        if (t.walk) t.cost = 1200.0 + waves * (double)max_stages * (stage + (b_pieces ? 20.0 * ((t.bn + 31) / 32 - 1) : 0.0)) + epilogue;
        if (best.grid == 0 || t.cost < best.cost) best = t;
        // the same tiles with a second launch
        const int tiles = m_count * t.n_tiles;
        t.splits = std::min(sms / tiles, min_stages / 4);
        t.grid = tiles * t.splits;
        const size_t bytes = (size_t)t.grid * BM * t.bn * sizeof(float);
        if (t.splits <= 1 || t.grid <= best.grid || bytes > partials_bytes) continue;
        t.second_launch = true;
        t.walk = false;
        t.cost = 1200.0 + (max_stages + t.splits - 1) / t.splits * (stage + 20.0 * (loads - 2 + (b_pieces ? (t.bn + 31) / 32 - 1 : 0))) + t.bn * 18.0 +
                 6500.0 + bytes / 2500.0;
        if (t.cost < best.cost) best = t;
    }
    return best;
}

// The divisors of conv_tc_kernel's work decoding; `p` is complete.
void set_divisors(Params& p, bool kernel_gradient)
{
    p.by_splits = FastDiv(p.splits);
    p.by_n_tiles = FastDiv(p.n_tiles);
    p.by_m_count = FastDiv(kernel_gradient ? p.m_tiles : p.tiles_w * p.tiles_h * p.tiles_n);
    p.by_tiles_w = FastDiv(p.tiles_w);
    p.by_tiles_h = FastDiv(p.tiles_h);
    p.by_kchunks = FastDiv(p.kchunks);
    p.by_kw = FastDiv(p.KW);
    p.by_sh = FastDiv(p.sh);
    p.by_sw = FastDiv(p.sw);
    p.pt_mod = p.pt % p.sh;
    p.pl_mod = p.pl % p.sw;
}

// False: the accumulators do not fit TMEM or the registers that take them over.
bool finish_plan(Plan& pl, bool kernel_gradient = false)
{
    Params& p = pl.p;
    const int b_stage = p.bn * BK * 4;
    const int per_stage = A_STAGE_BYTES + b_stage;
    if (p.x3) {
        // A and its residual take 64 TMEM columns per stage, what the accumulators (two and the small terms', or one of each
        // where two do not fit) leave; the residuals of B, which are made ahead of that, up to four tiles
        p.x3_slots = (512 - tmem_columns(kX3, p.bn, 0)) / 64;
        p.x3_slots = p.x3_slots >= 4 ? 4 : 2;   // powers of two
        p.x3_bslots = 4;
    }
    // two CTAs per SM when the grid has more CTAs than SMs, else one deep pipeline
    const bool half = pl.grid > sm_count() && p.bn <= kMaxSharedWidth && !p.x3;
    p.kind = p.x3 ? (p.bn <= kX3Width<kX3> ? kX3 : kX3Wide) : half ? kShared : p.bn <= 64 || p.mt > 1 ? kDual : p.splits == 1 ? kAlone : kShared;
    if (p.x3 && p.bn > kX3MaxWidth) return false;
    if (tmem_columns(p.kind, p.bn, p.x3_slots) > (half ? 256 : 512)) return false;
    if (p.walk) {
        p.stages = 8;
        while (walk_smem(p.stages, p.bn) > (size_t)kMaxSmem) --p.stages;
        pl.smem = walk_smem(p.stages, p.bn);
        p.skip_stage = -1;
        p.wait_cycles = kWaitCycles;
        set_divisors(p, kernel_gradient);
        return true;   // no scratch
    }
    const int budget = half ? (kMaxSmem / 2 - 2048) : (kMaxSmem - 2048);
    int stages = (budget - (p.x3 ? p.x3_bslots * b_stage : 0)) / per_stage;
    if (stages > 8) stages = 8;
    static const int forced_stages = env_int("DCG_TC_STAGES");
    if (forced_stages > 0 && forced_stages < stages) stages = forced_stages;
    if (stages < 2) stages = 2;
    // 3xTF32: the groups of warps tell the rounds of the ring apart with as many stages as groups or two more, and kX3Wide, which
    // looks once more, with one more, too.  So four stages for five at 112 and 128 columns, which is also quicker (a step of 64
    // images 3037 -> 2962 us, 128 -> 256 forward of 64 images 41.7 -> 39.6; five stages and that look 3071 to 3111, six with fewer residuals of B
    // 3343), and still four at 160 (kernel gradient of an RGB layer of 64 images 26.1 -> 26.2 us; three stages 29.4).
    if (p.x3) {
        const int groups = epilogue_groups(p.kind);
        if (stages < groups) return false;
        if (stages == groups + 1 && p.kind != kX3Wide) --stages;
    }
    if (p.kind == kDual) stages &= ~1;
    // the epilogue parks the 128 x bn tile (padded rows) and 128 row offsets in the (by then idle) stage ring
    while ((size_t)stages * per_stage < (size_t)kRedFloats(p.bn) * 4 + BM * 8) stages += p.kind == kDual ? 2 : 1;
    p.stages = stages;
    if (p.x3 && stages < 4) {   // a stage is released before its slot is used again
        p.x3_bslots = 2;
        p.x3_slots = 2;
    }
#ifdef DCG_TC_TRACING
    static const int debug = env_int("DCG_TC_DEBUG");
    p.debug = debug;
#endif
    pl.smem = (size_t)stages * per_stage + (p.x3 ? (size_t)p.x3_bslots * b_stage : 0) + 1024 /*alignment slack*/ + 24 * stages + 64;
    p.skip_stage = -1;
    p.wait_cycles = kWaitCycles;
    set_divisors(p, kernel_gradient);
    pl.partial_bytes = p.splits > 1 ? (size_t)pl.grid * BM * p.bn * sizeof(float) : 0;
    pl.ws_bytes = pl.partial_bytes;
    if (pl.xp_bytes || pl.k4_bytes) pl.ws_bytes = pl.k4_off() + align_up(pl.k4_bytes, 256);
    if (pl.ycol_bytes) pl.ws_bytes = pl.ycol_off() + align_up(pl.ycol_bytes, 256);
    return true;
}

// Padded-image geometry of a narrow-channel layer: rows s*i + di and columns s*j .. s*j + 7 of xp
// must exist for every output pixel and kernel row.
void narrow_geometry(const dcg_conv_desc& d, Plan& pl)
{
    pl.Hp = d.stride_h * (d.ho - 1) + d.kh;
    pl.Wp = (d.stride_w * (d.wo - 1) + 8 + 3) / 4 * 4;
    if (pl.Hp < d.h + d.pad_top) pl.Hp = d.h + d.pad_top;
    if (pl.Wp < d.w + d.pad_left) pl.Wp = (d.w + d.pad_left + 3) / 4 * 4;
    pl.xp_bytes = (size_t)d.n * pl.Hp * pl.Wp * 16;
}

// The channels of an MN-major operand lie in rows of 32 (one swizzle span).  A tensor map with the rows as a dimension of
// their own - one box per stage - exists for multiples of 32 only; other multiples of four are loaded row by row, the last
// one filled up with zeros.  The loads cost the producer more, but the CUDA cores, the other choice, take 5 to 15 times as
// long: 100 -> 132 forward, 3x3, of 8 images of 64 x 64 46 us for 645, 36 -> 100 kernel gradient, 5x5 / stride 2, of 16
// images of 40 x 40 21.5 for 130.  Below eight channels a tile holds too little, and 3xTF32 takes 10 us however small the
// layer is, which a few million products do not (12 -> 20, 3x3 / stride 2, of 4 images of 16 x 16: 10.4 and 6.4).
bool pieces_ok(const dcg_conv_desc& d, int channels)
{
    if (channels % 32 == 0) return true;
    const double products = (double)d.n * d.ho * d.wo * d.kh * d.kw * d.c * d.o;
    return channels % 4 == 0 && channels >= 8 && !(t_plan_x3 && products < 2e6);
}

int pad32(int channels) { return (channels + 31) / 32 * 32; }

bool narrow_ok(const dcg_conv_desc& d, double min_products)
{
    // Other output channels than multiples of 32: dy in pieces, the weights padded.  The repacks are a launch more, by the end
    // of which the CUDA cores are done with a small layer (3 -> 20 forward of 8 images of 32 x 32 6.7 us, 3 -> 180 of 4 of
    // 64 x 64 14 against 8); their kernel gradients take longest, for few outputs sum many pixels in order (3 -> 100, 5x5 /
    // stride 2, of 32 images of 96 x 96 402 us against 20, forward 142 against 26).
    const double products = (double)d.n * d.ho * d.wo * d.kh * d.kw * d.c * d.o;
    const bool o_ok = d.o % 32 == 0 || (d.o % 4 == 0 && d.o >= 8 && products >= min_products);
    return d.c <= 4 && d.kw <= 8 && o_ok && d.stride_h <= 8 && d.stride_w <= 8;
}

void base_params(Params& p, const dcg_conv_desc& d)
{
    p = Params{};
    p.x3 = t_plan_x3;
    p.N = d.n; p.H = d.h; p.W = d.w; p.C = d.c; p.KH = d.kh; p.KW = d.kw; p.O = d.o;
    p.Ho = d.ho; p.Wo = d.wo; p.sh = d.stride_h; p.sw = d.stride_w; p.pt = d.pad_top; p.pl = d.pad_left;
    p.m_tiles = 1; p.n_tiles = 1; p.splits = 1; p.kchunks = 1; p.mt = 1;
}

void use_tiling(Plan& pl, const Tiling& t)
{
    pl.p.bn = t.bn; pl.p.n_tiles = t.n_tiles; pl.p.splits = t.splits;
    pl.p.ext_finish = t.second_launch;
    pl.p.walk = t.walk;
    pl.grid = t.grid;
}

// `fit`: the tile follows the layer; the GEMM of a narrow-channel input gradient keeps 128 columns and power-of-two boxes, as
// the kernel with a resident B operand wants them.
bool plan_fwd(const dcg_conv_desc& d, Plan& pl, bool fit = true)
{
    const bool narrow = narrow_ok(d, 4e6);
    if (!narrow && (d.c % 4 != 0 || !pieces_ok(d, d.o) || d.stride_h > 8 || d.stride_w > 8)) return false;
    Params& p = pl.p;
    base_params(p, d);
    const bool pieces = !narrow && d.o % 32 != 0;
    if (pieces) { p.mt = 0; p.b_ch = d.o; }
    if (narrow || !fit) pixel_tile(BM, d.wo, d.ho, p.TW, p.TH, p.TN);
    else pixel_tile_fit(BM, d.wo, d.ho, d.n, d.stride_w, d.stride_h, false, p.TW, p.TH, p.TN);
    if (p.TW * d.stride_w > 256 || p.TH * d.stride_h > 256) return false;
    p.tiles_w = (d.wo + p.TW - 1) / p.TW; p.tiles_h = (d.ho + p.TH - 1) / p.TH; p.tiles_n = (d.n + p.TN - 1) / p.TN;
    p.kchunks = (d.c + BK - 1) / BK;
    const int m_count = p.tiles_w * p.tiles_h * p.tiles_n;
    if (narrow) {
        p.narrow = 1;
        p.kchunks = 1;
        narrow_geometry(d, pl);
        pl.k4_bytes = (size_t)d.kh * 32 * pad32(d.o) * sizeof(float);
    }
    const int stages = narrow ? d.kh : d.kh * d.kw * p.kchunks;
    if (narrow || !fit) {
        p.bn = d.o >= 128 ? 128 : pad32(d.o);
        p.n_tiles = (d.o + p.bn - 1) / p.bn;
        p.splits = choose_splits(m_count * p.n_tiles, stages);
        pl.grid = m_count * p.n_tiles * p.splits;
    } else {
        use_tiling(pl, choose_tiling(m_count, d.o, 32, stages, stages, 35, 2, pieces, 0, true));
    }
    return finish_plan(pl);
}

// The 1x1 FWD problem behind the DX of a narrow-channel layer: dy [n, ho, wo, o] times k2 [o][Jp].
dcg_conv_desc dx_gemm_desc(const dcg_conv_desc& d, int Jp)
{
    dcg_conv_desc g{};
    g.n = d.n; g.h = d.ho; g.w = d.wo; g.c = d.o; g.kh = 1; g.kw = 1; g.o = Jp; g.ho = d.ho; g.wo = d.wo;
    g.stride_h = 1; g.stride_w = 1; g.pad_top = 0; g.pad_left = 0;
    return g;
}

std::atomic<unsigned long long> g_dx_plans{0};
bool plan_dx(const dcg_conv_desc& d, Plan& pl)
{
    g_dx_plans.fetch_add(1, std::memory_order_relaxed);
    if (d.c <= 4 && d.o % 32 == 0 && d.stride_h <= d.kh && d.stride_w <= d.kw) {
        const int Jp = (d.kh * d.kw * 4 + 31) / 32 * 32;   // four columns per tap
        pl.Jp = Jp;
        pl.k2_bytes = (size_t)d.o * Jp * sizeof(float);
        pl.ycol_bytes = (size_t)d.n * d.ho * d.wo * Jp * sizeof(float);
        if (plan_fwd(dx_gemm_desc(d, Jp), pl, false)) {
            pl.p.planes = 1;
            pl.p.plane_stride = (unsigned long long)d.n * d.ho * d.wo * 4ull;
            pl.p.o_store = d.kh * d.kw * 4;   // the planes beyond the last tap are padding
            return true;
        }
        pl = Plan{};
    }
    if (d.o % 4 != 0 || d.stride_h > 8 || d.stride_w > 8) return false;
    if (d.stride_h > d.kh || d.stride_w > d.kw) return false;   // some parity class would have no tap
    Params& p = pl.p;
    base_params(p, d);
    const int ha = (d.h + d.stride_h - 1) / d.stride_h, wa = (d.w + d.stride_w - 1) / d.stride_w;
    pixel_tile_fit(BM, wa, ha, d.n, 1, 1, false, p.TW, p.TH, p.TN);
    p.tiles_w = (wa + p.TW - 1) / p.TW; p.tiles_h = (ha + p.TH - 1) / p.TH; p.tiles_n = (d.n + p.TN - 1) / p.TN;
    p.kchunks = (d.o + BK - 1) / BK;
    const int classes = d.stride_h * d.stride_w;
    const int min_taps = (d.kh / d.stride_h) * (d.kw / d.stride_w);
    const int max_taps = ((d.kh + d.stride_h - 1) / d.stride_h) * ((d.kw + d.stride_w - 1) / d.stride_w);
    use_tiling(pl, choose_tiling(classes * p.tiles_w * p.tiles_h * p.tiles_n, d.c, 16, (min_taps < 1 ? 1 : min_taps) * p.kchunks,
                                 max_taps * p.kchunks, 20, 2, false, 0, true));
    return finish_plan(pl);
}

// When the input gradient fuses its parity classes (conv_dxf_kernel): 0 never, 1 where one CTA per tile fills the
// GPU (default), 2 wherever the shape allows.  DCG_TC_DXF sets the default, dcg_debug_set_dx_mode overrides it.
std::atomic<int> g_dxf_mode{-1};
std::atomic<unsigned long long> g_dxf_launches{0};
int dxf_mode()
{
    static const int from_env = [] { const char* v = getenv("DCG_TC_DXF"); return v ? atoi(v) : 1; }();
    const int m = g_dxf_mode.load();
    return m >= 0 ? m : from_env;
}

// Keys are compared and hashed as bytes: they are zeroed before they are filled in.
template <typename Key>
struct BytesEqual {
    bool operator()(const Key& u, const Key& v) const { return std::memcmp(&u, &v, sizeof(Key)) == 0; }
};
template <typename Key>
struct BytesHash {
    size_t operator()(const Key& k) const
    {
        static_assert(sizeof(Key) % 4 == 0, "hashed by 32-bit words");
        uint32_t w[sizeof(Key) / 4];
        std::memcpy(w, &k, sizeof(Key));
        uint64_t h = 0xcbf29ce484222325ull;
        for (uint32_t v : w) h = (h ^ v) * 0x100000001b3ull;
        return (size_t)(h ^ (h >> 29));
    }
};

// A call without its tensors: what is known from the shape alone is kept per such key.
struct QueryKey {
    int dev, kind, x3;
    dcg_conv_desc d;
};
QueryKey query_key(const dcg_conv_desc& d, int kind, bool x3)
{
    QueryKey key;
    std::memset(&key, 0, sizeof(key));
    if (cudaGetDevice(&key.dev) != cudaSuccess) { cudaGetLastError(); key.dev = -1; }
    key.kind = kind; key.x3 = x3; key.d = d;
    return key;
}

// Whether the parity classes are quicker as tiles of their own, walked by persistent CTAs, than all of them together in `tiles`
// tiles of `bn` columns.  In clocks: a (class, tap) pair of a 32-channel chunk takes 233 of them at 64 columns and 297 at 128 in
// the class-fused kernel, a stage of the other one 300 at 128 columns and 512 at 256; a column of a class costs an epilogue 20,
// of which half of the shorter of loop and epilogue is hidden.  The class-fused tiles are four times as large, in boxes of powers
// of two and of at most 128 columns, which leaves much of them empty where the image, the channels or the last wave do not fit: 3 x 3 /
// stride 2, 192 -> 64, 30 images of 33 x 47 26.7 us fused, 13.4 apart; 192 -> 192, 32 images of 96 x 96 165 and 109.
// Where they fit, fused is quicker (5 x 5 / stride 2, 64 -> 128 of 64 images 15.6 and 21.0, 256 -> 512 of 512 images 69 and 81).
// The factor of 0.9 keeps the line on the safe side: of seventy layers drawn at random with twenty for which both are possible,
// apart is chosen for eighteen, all of them quicker so (0.39 to 0.98 of the fused time), and not for two that would take 0.84 and 0.87.
bool classes_apart_modelled(const dcg_conv_desc& d, int tiles, int bn, int ncls)
{
    Plan apart;
    if (!plan_dx(d, apart) || !apart.p.walk) return false;
    const Params& p = apart.p;
    const double sms = sm_count(), pairs = (double)d.kh * d.kw * ((d.o + BK - 1) / BK);
    auto both = [](double loop, double epilogue) { return std::max(loop, epilogue) + 0.5 * std::min(loop, epilogue); };
    const double fused = std::ceil(tiles / sms) * both(pairs * (bn <= 64 ? 233.0 : 169.0 + bn), 20.0 * ncls * bn);
    const double stage = p.bn > 128 ? 300.0 + (p.bn - 128) * (212.0 / 128) : 300.0;
    const double mine = both((double)p.tiles_w * p.tiles_h * p.tiles_n * p.n_tiles * pairs / sms * stage, std::ceil(apart.grid / sms) * 20.0 * p.bn) +
                        0.5 * stage * pairs / ncls;   // (the classes differ in length)
    return mine < 0.9 * fused;
}

// The same, kept: a call on new addresses is planned again, and this is a second plan (host time of an input gradient with new
// addresses every time: 64 images of 32 x 32, 64 -> 128 9.1 -> 5.8 us; 20 of 33 x 47, 192 -> 64, classes apart 11.9 -> 7.5).
bool classes_apart_quicker(const dcg_conv_desc& d, int tiles, int bn, int ncls)
{
    static std::mutex mutex;
    static std::unordered_map<QueryKey, bool, BytesHash<QueryKey>, BytesEqual<QueryKey>> known;
    const QueryKey key = query_key(d, kConvDx, false);
    {
        std::lock_guard<std::mutex> lock(mutex);
        const auto it = known.find(key);
        if (it != known.end()) return it->second;
    }
    const bool quicker = classes_apart_modelled(d, tiles, bn, ncls);
    std::lock_guard<std::mutex> lock(mutex);
    if (known.size() >= 4096) known.clear();
    return known[key] = quicker;
}

// The class-fused input gradient (conv_dxf_kernel): windows of dy, the (class, tap) pairs that read each, and
// the order of both.
bool plan_dxf(const dcg_conv_desc& d, Plan& pl, CfTable& t)
{
    const int mode = dxf_mode();
    if (mode == 0 || t_plan_x3) return false;
    if (d.o % 4 != 0) return false;   // rows of dy and of the weights are 16-byte aligned for TMA
    // <= 4 input channels: a tile is 18 short stages and four element-wise epilogues - measured at 46 us against
    // 25 us for GEMM + gather on the 3-channel layer at batch 64 (one CTA per SM has nothing to hide its set-up behind)
    if (d.c <= 4) return false;
    if (d.stride_h > d.kh || d.stride_w > d.kw) return false;
    const int ncls = d.stride_h * d.stride_w;
    if (ncls < 2 || ncls > 4) return false;
    Params& p = pl.p;
    base_params(p, d);
    const int ha = (d.h + d.stride_h - 1) / d.stride_h, wa = (d.w + d.stride_w - 1) / d.stride_w;
    pixel_tile(BM, wa, ha, p.TW, p.TH, p.TN);
    p.tiles_w = (wa + p.TW - 1) / p.TW; p.tiles_h = (ha + p.TH - 1) / p.TH; p.tiles_n = (d.n + p.TN - 1) / p.TN;
    int bn = (d.c + 15) / 16 * 16;
    if (bn > 128) bn = 128;
    if (ncls * bn > 512) return false;
    p.bn = bn;
    p.n_tiles = (d.c + bn - 1) / bn;
    p.kchunks = (d.o + BK - 1) / BK;
    const int tiles = p.tiles_w * p.tiles_h * p.tiles_n * p.n_tiles;
    // one CTA per tile, no K partitions: only where the tiles alone fill (most of) the GPU
    if (mode != 2 && tiles * 4 < sm_count() * 3) return false;
    if (mode == 1 && classes_apart_quicker(d, tiles, bn, ncls)) return false;
    // every (class, tap) pair with the window it reads
    struct Pair { int sy, sx, cls, kh, kw; };
    std::vector<Pair> pairs;
    for (int ph = 0; ph < d.stride_h; ++ph)
        for (int pw = 0; pw < d.stride_w; ++pw) {
            const int rh = (ph + d.pad_top) % d.stride_h, eh = (ph + d.pad_top) / d.stride_h;
            const int rw = (pw + d.pad_left) % d.stride_w, ew = (pw + d.pad_left) / d.stride_w;
            for (int a = 0; rh + d.stride_h * a < d.kh; ++a)
                for (int b = 0; rw + d.stride_w * b < d.kw; ++b)
                    pairs.push_back({eh - a, ew - b, ph * d.stride_w + pw, rh + d.stride_h * a, rw + d.stride_w * b});
        }
    // classes in the order "fewest windows still to fetch first"; the windows follow that order
    t = CfTable{};
    t.ncls = ncls;
    std::vector<std::pair<int, int>> wins;   // scheduled windows
    auto scheduled = [&](int sy, int sx) {
        for (auto& w : wins) if (w.first == sy && w.second == sx) return true;
        return false;
    };
    bool finished[4] = {false, false, false, false};
    for (int ci = 0; ci < ncls; ++ci) {
        int best = -1, best_need = 1 << 30;
        for (int c = 0; c < ncls; ++c) {
            if (finished[c]) continue;
            std::vector<std::pair<int, int>> need;
            for (auto& q : pairs)
                if (q.cls == c && !scheduled(q.sy, q.sx)) {
                    bool seen = false;
                    for (auto& n : need) seen |= n.first == q.sy && n.second == q.sx;
                    if (!seen) need.push_back({q.sy, q.sx});
                }
            if ((int)need.size() < best_need) { best_need = (int)need.size(); best = c; }
        }
        if (best < 0) return false;
        bool any = false;
        for (auto& q : pairs)
            if (q.cls == best) {
                any = true;
                if (!scheduled(q.sy, q.sx)) wins.push_back({q.sy, q.sx});
            }
        if (!any) return false;   // a class without taps
        finished[best] = true;
        t.order[ci] = best;
    }
    // stages: a window with its pairs, at most pb per stage (about 48 KB)
    const int b_tile = bn * BK * 4;
    int pb = (48 * 1024 - A_STAGE_BYTES) / b_tile;
    if (pb > 4) pb = 4;
    if (pb < 1) pb = 1;
    // TMEM order of the classes: for 2 x 2 classes the cyclic order (0,0) (0,1) (1,1) (1,0), in which the classes
    // of one row / one column parity are neighbours, so that the pairs of a window merge into wide MMAs
    for (int c = 0; c < ncls; ++c) t.slot_of_class[c] = c;
    if (d.stride_h == 2 && d.stride_w == 2) { t.slot_of_class[2] = 3; t.slot_of_class[3] = 2; }
    int last_stage[4] = {-1, -1, -1, -1};
    bool started[4] = {false, false, false, false};
    int ns = 0, max_units = 0;
    for (size_t w = 0; w < wins.size(); ++w) {
        if (wins[w].first < -128 || wins[w].first > 127 || wins[w].second < -128 || wins[w].second > 127) return false;
        // the pairs of this window in TMEM order
        std::vector<Pair> mine;
        for (auto& q : pairs)
            if (q.sy == wins[w].first && q.sx == wins[w].second) mine.push_back(q);
        for (size_t a = 0; a < mine.size(); ++a)
            for (size_t b = a + 1; b < mine.size(); ++b)
                if (t.slot_of_class[mine[b].cls] < t.slot_of_class[mine[a].cls]) std::swap(mine[a], mine[b]);
        for (size_t first = 0; first < mine.size(); first += pb) {
            if (ns == 32) return false;
            CfWin& cw = t.win[ns];
            cw.sy = (signed char)wins[w].first; cw.sx = (signed char)wins[w].second;
            const size_t end = std::min(mine.size(), first + (size_t)pb);
            for (size_t a = first; a < end; ++a) {
                const Pair& q = mine[a];
                const int slot = t.slot_of_class[q.cls];
                const int fresh = started[q.cls] ? 0 : 1;
                cw.kh[cw.n] = (unsigned char)q.kh; cw.kw[cw.n] = (unsigned char)q.kw;
                // joins the running MMA if its accumulator follows directly, starts the same way and N stays <= 256
                CfRun* run = cw.runs > 0 ? &cw.run[cw.runs - 1] : nullptr;
                if (run && run->slot + run->count == slot && run->fresh == fresh && (run->count + 1) * bn <= 256) ++run->count;
                else cw.run[cw.runs++] = {1, (unsigned char)slot, cw.n, (unsigned char)fresh};
                last_stage[q.cls] = ns;
                ++cw.n;
            }
            for (size_t a = first; a < end; ++a) started[mine[a].cls] = true;
            cw.units = (unsigned char)((A_STAGE_BYTES + cw.n * b_tile + kCfUnit - 1) / kCfUnit);
            if (cw.units > max_units) max_units = cw.units;
            ++ns;
        }
    }
    t.nwin = ns;
    for (int c = 0; c < ncls; ++c) {
        if (last_stage[c] < 0) return false;
        t.win[last_stage[c]].last |= (unsigned char)(1u << c);
    }
    p.splits = 1;
    pl.grid = tiles;
    const int fixed = 1024 + kCfEpi / 32 * kCfPatch + 16 * kCfBars + 64;
    int units = (kMaxSmem - fixed) / kCfUnit;
    if (units > kCfMaxUnits) units = kCfMaxUnits;
    if (units < 3 * max_units) return false;   // three stages in flight
    p.stages = units;
    pl.smem = (size_t)units * kCfUnit + fixed;
    p.skip_stage = -1;
    p.wait_cycles = kWaitCycles;
    set_divisors(p, false);
    pl.partial_bytes = 0;
    pl.ws_bytes = 0;
    return true;
}

bool plan_dk(const dcg_conv_desc& d, Plan& pl, size_t ws_bytes)
{
    const bool narrow = narrow_ok(d, 4e5);
    if (!narrow && (!pieces_ok(d, d.c) || !pieces_ok(d, d.o) || d.stride_h > 8 || d.stride_w > 8)) return false;
    Params& p = pl.p;
    base_params(p, d);
    const bool pieces = !narrow && (d.c % 32 != 0 || d.o % 32 != 0);
    pixel_tile_fit(BK, d.wo, d.ho, d.n, d.stride_w, d.stride_h, true, p.TW, p.TH, p.TN);   // 32 output pixels per K stage
    if (p.TW * d.stride_w > 256 || p.TH * d.stride_h > 256) return false;
    p.tiles_w = (d.wo + p.TW - 1) / p.TW; p.tiles_h = (d.ho + p.TH - 1) / p.TH; p.tiles_n = (d.n + p.TN - 1) / p.TN;
    if (narrow) {
        // rows = output channels (from dy), columns = 32 window slots per kernel row: one tile holds
        // all of dk, so dy is read exactly once; the parallelism comes from partitioning the pixels
        // over about as many CTAs as there are SMs, whose partial tiles a second kernel adds up.
        // 3xTF32 of seven or eight kernel rows, which are wider than it can sum, takes two tiles of four
        if (d.kh * 32 > 256) return false;
        p.narrow = 1;
        p.swap = 1;
        if (d.o % 32 != 0) { p.mt = 0; p.a_ch = d.o; }
        p.m_tiles = (d.o + BM - 1) / BM;
        const int rows = p.x3 && 32 * d.kh > kX3MaxWidth ? (d.kh + 1) / 2 : d.kh;
        p.bn = 32 * rows;
        p.n_tiles = (d.kh + rows - 1) / rows;
        narrow_geometry(d, pl);
        const int k_stages = p.tiles_w * p.tiles_h * p.tiles_n;
        int parts = sm_count() / (p.m_tiles * p.n_tiles);
        if (parts > k_stages / 4) parts = k_stages / 4;   // at least 4 K stages per CTA
        if (parts < 1) parts = 1;
        p.splits = parts;
        p.ext_finish = parts > 1 ? 1 : 0;
        pl.grid = p.m_tiles * p.n_tiles * p.splits;
        return finish_plan(pl, true);
    }
    // M (128 accumulator rows) is the input-channel axis, so that dk rows are contiguous along the accumulator columns,
    // with the channels of four or two taps on top of one another where there are only 32 or 64 of them; or M is the
    // output-channel axis, where that is quicker.
    const int stages = p.tiles_w * p.tiles_h * p.tiles_n, taps = d.kh * d.kw;
    const int mt = pieces ? 1 : d.c == 64 && taps >= 2 ? 2 : d.c == 32 && taps >= 4 ? 4 : 1;
    const int rows_c = (d.c + BM - 1) / BM, rows_o = (d.o + BM - 1) / BM;
    static const int roles = env_int("DCG_TC_ROLES");
    auto row_pieces = [&](int ch) { return pieces ? (ch < BM ? (ch + 31) / 32 : BM / 32) - 1 : 0; };
    const Tiling plain = choose_tiling((taps + mt - 1) / mt * rows_c, d.o, 32, stages, stages, 20, 1 + mt + row_pieces(d.c), pieces, ws_bytes);
    const Tiling swapped = choose_tiling(taps * rows_o, d.c, 32, stages, stages, 30, 2 + row_pieces(d.o), pieces, ws_bytes);
    p.swap = roles ? roles == 2 : swapped.cost < plain.cost;
    p.m_tiles = p.swap ? rows_o : rows_c;
    p.mt = p.swap ? 1 : mt;
    if (pieces) { p.mt = 0; p.a_ch = p.swap ? d.o : d.c; p.b_ch = p.swap ? d.c : d.o; }
    use_tiling(pl, p.swap ? swapped : plain);
    return finish_plan(pl, true);
}

// The forward of a <= 4-channel layer from its image (conv_fwd_rgb_kernel): all output channels in one tile, everything it keeps
// in shared memory.  It needs no scratch and is the quicker one at every size measured; the weights' rows have to be TMA rows.
bool plan_rgb(const dcg_conv_desc& d, Plan& pl, RgbArgs& g)
{
    if (t_plan_x3 || d.c > 4 || d.o % 32 != 0 || d.o > 128 || d.kw > 8 || d.kh * (d.kw * d.c <= 16 ? 16 : 32) > kRgbMaxChunks * BK) return false;
    Params& p = pl.p;
    base_params(p, d);
    pixel_tile(BM, d.wo, d.ho, p.TW, p.TH, p.TN);
    p.tiles_w = (d.wo + p.TW - 1) / p.TW; p.tiles_h = (d.ho + p.TH - 1) / p.TH; p.tiles_n = (d.n + p.TN - 1) / p.TN;
    p.bn = d.o;
    p.stages = 2;
    p.skip_stage = -1;
    p.wait_cycles = kWaitCycles;
    set_divisors(p, false);
    g.kwc = d.kw * d.c;
    const int places = g.kwc <= 16 ? 16 : 32;
    g.chunks = (d.kh * places + BK - 1) / BK;
    g.ksteps = d.kh * places / 8;
    const long long rows = (long long)p.TN * ((p.TH - 1) * d.stride_h + d.kh), row_len = ((long long)(p.TW - 1) * d.stride_w + d.kw) * d.c;
    if (rows * row_len * 4 > kMaxSmem) return false;
    g.rows = (int)rows; g.row_len = (int)row_len;
    // image rows of whole 16 bytes: a patch is one box of (row, rows, images)
    const int box = (int)align_up(row_len + 3, 4);
    g.tma = d.w * d.c % 4 == 0 && box <= 256 && (p.TH - 1) * d.stride_h + d.kh <= 256;
    g.pitch = g.tma ? box : (g.row_len + 1) & ~1;
    g.patch_tx = (unsigned)(rows * g.pitch * 4);
    g.patch_bytes = (int)align_up((rows * g.pitch + places + 4) * 4, 128);   // (the last pixel's places end beyond its row)
    g.tiles = p.tiles_w * p.tiles_h * p.tiles_n;
    pl.grid = g.tiles < sm_count() ? g.tiles : sm_count();
    for (g.patches = 4; g.patches >= 2; --g.patches) {
        pl.smem = rgb_smem(g.chunks, p.bn, (size_t)g.patches * g.patch_bytes);
        if (pl.smem <= (size_t)kMaxSmem) return true;
    }
    return false;
}

// `ws_bytes`: scratch that there is, as far as a plan may do with less.
bool make_plan(const dcg_conv_desc& d, int kind, Plan& pl, size_t ws_bytes = (size_t)-1)
{
    RgbArgs rgb;
    switch (kind) {
    case kConvFwd:
        if (plan_rgb(d, pl, rgb)) return true;
        pl = Plan{};
        return plan_fwd(d, pl);
    case kConvDx: return plan_dx(d, pl);
    case kConvDk: return plan_dk(d, pl, ws_bytes);
    default: return false;
    }
}

// Testing hooks (dcg_debug_set_wait_limit / dcg_debug_skip_stage): the wait limit of every barrier
// wait in SM clocks, and a pipeline stage the producer leaves out so that a wait runs into that limit.
long long default_wait_cycles()
{
    const char* v = getenv("DCG_TC_WAIT_CYCLES");   // experiments: a shorter limit than the ~1 s default
    const long long c = v ? atoll(v) : 0;
    return c > 0 ? c : kWaitCycles;
}
std::atomic<long long> g_wait_cycles{default_wait_cycles()};
std::atomic<int> g_test_skip_stage{-1};

template <int MODE>
int launch_grid(const CUtensorMap& ma, const CUtensorMap& mb, const Params& p, int grid, size_t smem, cudaStream_t stream)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)(64 + 128 * epilogue_groups(p.kind)));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    static const int no_pdl = env_int("DCG_TC_NO_PDL");
    if (!no_pdl) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    if (p.splits > 1 && !p.ext_finish) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = (unsigned)p.splits;   // blockIdx.x = tile * splits + split: one cluster per tile
        attr[na].val.clusterDim.y = 1;
        attr[na].val.clusterDim.z = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    using Kernel = void (*)(CUtensorMap, CUtensorMap, Params);
    // (only the kernel gradient of an RGB layer is wider than 128 columns in 3xTF32)
    static const Kernel kernels[] = {conv_tc_kernel<MODE, kShared>, conv_tc_kernel<MODE, kX3>, conv_tc_kernel<MODE, kAlone>,
                                     conv_tc_kernel<MODE, kDual>};
    int form = 0;
    Kernel kernel = p.kind == kX3Wide ? nullptr : kernels[p.kind];
    if constexpr (MODE != MODE_DX) {
        static const Kernel pieces[] = {conv_tc_kernel<MODE, kShared, 0>, conv_tc_kernel<MODE, kX3, 0>, conv_tc_kernel<MODE, kAlone, 0>,
                                        conv_tc_kernel<MODE, kDual, 0>};
        if (p.mt == 0 && p.kind != kX3Wide) { form = 1; kernel = pieces[p.kind]; }
    }
    if constexpr (MODE == MODE_DK) {
        if (p.kind == kX3Wide) { form = p.mt == 0; kernel = p.mt == 0 ? conv_tc_kernel<MODE_DK, kX3Wide, 0> : conv_tc_kernel<MODE_DK, kX3Wide>; }
    }
    if (!kernel) return fail(DCG_ERR_UNSUPPORTED, "conv_tc_kernel: no kernel of %d columns for this operator", p.bn);
    if constexpr (MODE == MODE_DK) {
        static const Kernel more_taps[2][4] = {
            {conv_tc_kernel<MODE_DK, kShared, 2>, conv_tc_kernel<MODE_DK, kX3, 2>, nullptr, conv_tc_kernel<MODE_DK, kDual, 2>},
            {conv_tc_kernel<MODE_DK, kShared, 4>, conv_tc_kernel<MODE_DK, kX3, 4>, nullptr, conv_tc_kernel<MODE_DK, kDual, 4>}};
        if (p.mt > 1) { form = 2 + p.mt / 4; kernel = more_taps[p.mt / 4][p.kind]; }
    }
    // each form is loaded when it is first needed, not all of them with the first convolution
    static OncePerDevice once[4][kKinds];
    DCG_CUDA(allow_smem(once[form][p.kind], kernel, kMaxSmem));
    const cudaError_t err = cudaLaunchKernelEx(&cfg, kernel, ma, mb, p);
    if (err != cudaSuccess) return fail(DCG_ERR_CUDA, "conv_tc_kernel launch: %s", cudaGetErrorString(err));
    count_launch();
    return DCG_OK;
}

template <int MODE>
int launch_walk(const CUtensorMap& ma, const CUtensorMap& mb, const Plan& pl, cudaStream_t stream)
{
    using Kernel = void (*)(CUtensorMap, CUtensorMap, Params, int);
    static const Kernel kernels[2] = {conv_tc_walk_kernel<MODE>, conv_tc_walk_kernel<MODE, MODE == MODE_FWD>};
    static OncePerDevice once[2];
    const int pieces = pl.p.mt == 0;
    DCG_CUDA(allow_smem(once[pieces], kernels[pieces], kMaxSmem));
    launch_pdl(kernels[pieces], (unsigned)std::min(pl.grid, sm_count()), kWalkThreads, pl.smem, stream, ma, mb, pl.p, pl.grid);
    DCG_LAUNCH_CHECK("conv_tc_walk_kernel");
    return DCG_OK;
}

template <int MODE>
int launch(const CUtensorMap& ma, const CUtensorMap& mb, Plan& pl, float* out, const EpilogueArgs& ep,
           int channels, void* ws, size_t ws_bytes, cudaStream_t stream)
{
    Params& p = pl.p;
    p.out = out;
    p.ep = ep;
    p.scratch = nullptr;
    p.skip_stage = g_test_skip_stage.load();
    p.wait_cycles = g_wait_cycles.load();
    if (p.splits > 1) {
        if (!ws || ws_bytes < pl.ws_bytes)
            return fail(DCG_ERR_WORKSPACE, "conv (tensor path): workspace %zu < %zu bytes", ws_bytes, pl.ws_bytes);
        p.scratch = static_cast<float*>(ws);
    }
    (void)channels;
    if constexpr (MODE != MODE_DK)
        if (p.walk) return launch_walk<MODE>(ma, mb, pl, stream);
    const int st = launch_grid<MODE>(ma, mb, p, pl.grid, pl.smem, stream);
    if (st) return st;
    if (p.ext_finish && !p.narrow) {
        const dim3 fgrid((unsigned)(pl.grid / p.splits), (unsigned)(BM / kFinishRows * (p.bn / kFinishCols)));
        launch_pdl(p.swap ? dk_finish_kernel<true> : dk_finish_kernel<false>, fgrid, 256, 0, stream, p.scratch, out, p.splits, p.bn, p.n_tiles,
                   p.m_tiles, p.mt > 1 ? p.mt : 1, p.KH * p.KW, p.C, p.O);
        DCG_LAUNCH_CHECK("dk_finish_kernel");
    } else if (p.ext_finish) {
        const dim3 fgrid((unsigned)(p.bn * p.n_tiles), (unsigned)((p.O + 31) / 32));
        launch_pdl(dk_narrow_finish_kernel, fgrid, 256, 0, stream, p.scratch, out, p.splits, p.bn, p.n_tiles, p.KH, p.KW, p.C, p.O);
        DCG_LAUNCH_CHECK("dk_narrow_finish_kernel");
    }
    return DCG_OK;
}

struct Prepared;
int launch_dxf(Prepared& pr, float* out, const EpilogueArgs& ep, cudaStream_t stream);
bool short_ok(const Plan& pl);
int launch_short(Prepared& pr, bool narrow, float* out, const EpilogueArgs& ep, cudaStream_t stream);
int launch_dx3(Prepared& pr, float* out, const EpilogueArgs& ep, cudaStream_t stream);

// Narrow-channel layers: builds the padded 4-channel image (and, for FWD, the repacked weights) in
// the caller's scratch and returns their addresses.
int narrow_prepare(const dcg_conv_desc& d, const Plan& pl, const float* x, const float* k, void* ws, size_t ws_bytes,
                   cudaStream_t stream, float** xp_out, float** k4_out)
{
    if (!ws || ws_bytes < pl.ws_bytes)
        return fail(DCG_ERR_WORKSPACE, "conv (tensor path, narrow input): workspace %zu < %zu bytes", ws_bytes, pl.ws_bytes);
    uint8_t* base = static_cast<uint8_t*>(ws);
    float* xp = reinterpret_cast<float*>(base + pl.xp_off());
    const size_t pixels = (size_t)d.n * pl.Hp * pl.Wp;
    size_t blocks = (pixels + 255) / 256;
    const size_t cap = (size_t)sm_count() * 16;
    if (blocks > cap) blocks = cap;
    *xp_out = xp;
    if (k4_out) {   // forward: image and weights in one launch
        float* k4 = reinterpret_cast<float*>(base + pl.k4_off());
        const int total = d.kh * 32 * pad32(d.o);
        const int k4_blocks = (total + 255) / 256;
        launch_pdl(repack_narrow_k4_kernel, (unsigned)(blocks + k4_blocks), 256, 0, stream, x, reinterpret_cast<float4*>(xp),
                   d.n, d.h, d.w, d.c, pl.Hp, pl.Wp, d.pad_top, d.pad_left, k, k4, d.kh, d.kw, d.o, pad32(d.o), k4_blocks);
        DCG_LAUNCH_CHECK("repack_narrow_k4_kernel");
        *k4_out = k4;
    } else {
        launch_pdl(repack_narrow_kernel, (unsigned)blocks, 256, 0, stream, x, reinterpret_cast<float4*>(xp), d.n, d.h, d.w,
                   d.c, pl.Hp, pl.Wp, d.pad_top, d.pad_left);
        DCG_LAUNCH_CHECK("repack_narrow_kernel");
    }
    return DCG_OK;
}

// The overlapping-window view of xp [n][Hp][Wp][4]: (32 floats, j, i, n, kernel row) where output
// pixel (i, j) and kernel row r address xp[n][s*i + r][s*j][0].  Box (32, tw, th, tn, rows).
int map_window(CUtensorMap* map, const float* xp, const dcg_conv_desc& d, const Plan& pl, int tw, int th, int tn,
               bool mn_major, int rows)
{
    const cuuint64_t row = (cuuint64_t)pl.Wp * 16;
    const cuuint64_t dims[5] = {32, (cuuint64_t)d.wo, (cuuint64_t)d.ho, (cuuint64_t)d.n, (cuuint64_t)d.kh};
    const cuuint64_t strides[4] = {(cuuint64_t)d.stride_w * 16, (cuuint64_t)d.stride_h * row, (cuuint64_t)pl.Hp * row, row};
    const cuuint32_t box[5] = {32, (cuuint32_t)tw, (cuuint32_t)th, (cuuint32_t)tn, (cuuint32_t)rows};
    const cuuint32_t es[5] = {1, 1, 1, 1, 1};
    return encode_map(map, xp, 5, dims, mn_major, strides, box, es);
}

// ---- prepared calls: plan + tensor maps, cached ------------------------------------------------------
// Planning a convolution and encoding its two tensor maps costs the host ~10 us.  A training step
// or the reference's Graph::run issues the same convolutions on the same buffers over and over, so
// the result is kept per (device, operator, shape, operand addresses, scratch address, precision)
// in a small table; a hit leaves only the launch.
// What an RGB forward writes and its gate: output, raw result, pre-activation, gate.  They are no part of the key.
struct RgbMaps {
    const void* of[4];   // the tensor that a map is of (null: none yet)
    CUtensorMap map[4];
};
struct Prepared {
    Plan pl;
    CUtensorMap ma, mb;
    bool dxf = false;   // input gradient with the parity classes fused (conv_dxf_kernel); cf is its table
    union {
        CfTable cf;
        RgbMaps rgb_maps;   // rgb
    };
    bool dx3 = false;   // input gradient of a <= 4-channel layer as one GEMM + gather kernel (conv_dx3_kernel)
    Dx3Args dx3_args;
    bool rgb = false;   // forward of a <= 4-channel layer from its image (conv_fwd_rgb_kernel)
    RgbArgs rgb_args;
    Prepared() { std::memset(&rgb_maps, 0, sizeof(rgb_maps)); }
};

int launch_dxf(Prepared& pr, float* out, const EpilogueArgs& ep, cudaStream_t stream)
{
    static OncePerDevice once;
    DCG_CUDA(allow_smem(once, conv_dxf_kernel, kMaxSmem));
    Params& p = pr.pl.p;
    p.out = out;
    p.ep = ep;
    p.scratch = nullptr;
    p.wait_cycles = g_wait_cycles.load();
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)pr.pl.grid);
    cfg.blockDim = dim3(kCfThreads);
    cfg.dynamicSmemBytes = pr.pl.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    int na = 0;
    static const int no_pdl = env_int("DCG_TC_NO_PDL");
    if (!no_pdl) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    const cudaError_t err = cudaLaunchKernelEx(&cfg, conv_dxf_kernel, pr.ma, pr.mb, p, pr.cf);
    if (err != cudaSuccess) return fail(DCG_ERR_CUDA, "conv_dxf_kernel launch: %s", cudaGetErrorString(err));
    count_launch();
    g_dxf_launches.fetch_add(1);
    return DCG_OK;
}

// Whether a forward plan goes to the persistent short-K kernel: a single column tile, no K partitions, weights
// that fit the resident area, more tiles than SMs (else there is nothing to walk).  DCG_TC_SHORT=0 switches it off.
bool short_ok(const Plan& pl)
{
    static const int off = [] { const char* v = getenv("DCG_TC_SHORT"); return v && atoi(v) == 0 ? 1 : 0; }();
    const Params& p = pl.p;
    if (off || p.x3 || p.splits != 1 || p.n_tiles != 1 || p.bn > 128 || p.bn % 32 != 0 || p.TW * p.TH * p.TN != BM) return false;
    const int ksteps = p.narrow ? p.KH : p.KH * p.KW * p.kchunks;
    if (!p.narrow && (p.KH != 1 || p.KW != 1 || !p.planes)) return false;   // the GEMM of the 3-channel input gradient
    if (p.narrow && (p.planes || p.O % 32 != 0)) return false;
    if (ksteps < 1 || ksteps * p.bn * BK * 4 > kShortMaxB) return false;
    return pl.grid > sm_count();
}

int launch_short(Prepared& pr, bool narrow, float* out, const EpilogueArgs& ep, cudaStream_t stream)
{
    static OncePerDevice once[2];
    DCG_CUDA(allow_smem(once[narrow], narrow ? conv_fwd_short_kernel<true> : conv_fwd_short_kernel<false>, kMaxSmem / 2));
    Params& p = pr.pl.p;
    p.out = out;
    p.ep = ep;
    p.scratch = nullptr;
    p.wait_cycles = g_wait_cycles.load();
    const int tiles = pr.pl.grid;
    const int ksteps = narrow ? p.KH : p.kchunks;
    int grid = 2 * sm_count();
    if (grid > tiles) grid = tiles;
    p.stages = narrow ? 3 : kShortMaxStages;
    const size_t smem = 1024 + (size_t)ksteps * p.bn * BK * 4 + (size_t)p.stages * A_STAGE_BYTES +
                        (narrow ? (size_t)(kEpi / 32) * kPatchBytes : 0) + 16 * kShortMaxStages + 64;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    int na = 0;
    static const int no_pdl = env_int("DCG_TC_NO_PDL");
    if (!no_pdl) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    const cudaError_t err = narrow ? cudaLaunchKernelEx(&cfg, conv_fwd_short_kernel<true>, pr.ma, pr.mb, p, tiles, ksteps)
                                   : cudaLaunchKernelEx(&cfg, conv_fwd_short_kernel<false>, pr.ma, pr.mb, p, tiles, ksteps);
    if (err != cudaSuccess) return fail(DCG_ERR_CUDA, "conv_fwd_short_kernel launch: %s", cudaGetErrorString(err));
    count_launch();
    return DCG_OK;
}

// GEMM + gather in one kernel for the input gradient of a <= 4-channel layer (conv_dx3_kernel): stride 2, at most
// 32 taps, dy rows of at most 32 pixels and at most 64 channels (the resident weights and the products of a tile
// share the CTA's shared memory).  DCG_TC_DX3=0 switches it off.
bool plan_dx3(const dcg_conv_desc& d, Plan& pl, Dx3Args& g)
{
    static const int off = [] { const char* v = getenv("DCG_TC_DX3"); return v && atoi(v) == 0 ? 1 : 0; }();
    if (off || t_plan_x3) return false;
    if (d.c > 4 || d.stride_h != 2 || d.stride_w != 2 || d.kh * d.kw > 32 || d.kh < 2 || d.kw < 2) return false;
    if (d.o % 32 != 0 || d.o > 64 || d.wo > 32 || d.pad_top >= d.kh || d.pad_left >= d.kw) return false;
    // the most output rows (2R) whose contributing dy rows fit the 8 rows of a tile, but no more than it takes to give every SM
    // a tile: the gather of a tile is what a small batch waits for (one image 6.7 us as 32 tiles of two rows, 9.0 as 6 of 12)
    int R = 0, lo = 0;
    const int tiles_each = sm_count() / d.n > 1 ? sm_count() / d.n : 1, rows = (d.h + 1) / 2;
    int widest = (rows + tiles_each - 1) / tiles_each;
    if (widest > kDx3Rows) widest = kDx3Rows;
    for (int r = widest; r >= 1 && R == 0; --r) {
        int mn = 1 << 30, mx = -(1 << 30);
        for (int hl = 0; hl < 2 * r; ++hl)
            for (int di = (hl + d.pad_top) & 1; di < d.kh; di += 2) {
                const int v = hl + d.pad_top - di;
                const int i = v >= 0 ? v / 2 : -((-v + 1) / 2);   // floor
                if (i < mn) mn = i;
                if (i > mx) mx = i;
            }
        if (mx - mn + 1 <= kDx3Rows) { R = r; lo = mn; g.mts = (mx - mn + 4) / 4; }
    }
    if (R == 0) return false;
    Params& p = pl.p;
    base_params(p, d);
    p.kchunks = d.o / BK;
    p.bn = 128;
    p.splits = 1;
    p.skip_stage = -1;
    p.wait_cycles = kWaitCycles;
    g.R = R;
    g.lo = lo;
    g.tiles_per_img = (d.h + 2 * R - 1) / (2 * R);
    g.tiles = d.n * g.tiles_per_img;
    g.by_tiles_per_img = FastDiv(g.tiles_per_img);
    pl.grid = g.tiles < sm_count() ? g.tiles : sm_count();
    pl.smem = 1024 + (size_t)p.kchunks * 128 * BK * 4 + (size_t)kDx3Stages * A_STAGE_BYTES +
              (size_t)d.kh * d.kw * kDx3Rows * 32 * 16 + 16 * kDx3Stages + 64;
    pl.ws_bytes = 0;
    return pl.smem <= (size_t)kMaxSmem;
}

int launch_dx3(Prepared& pr, float* out, const EpilogueArgs& ep, cudaStream_t stream)
{
    Params& p = pr.pl.p;
    const bool five = p.KH == 5 && p.KW == 5;
    static OncePerDevice once[2];
    DCG_CUDA(allow_smem(once[five], five ? conv_dx3_kernel<5, 5> : conv_dx3_kernel<0, 0>, kMaxSmem));
    p.out = out;
    p.ep = ep;
    p.scratch = nullptr;
    p.wait_cycles = g_wait_cycles.load();
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)pr.pl.grid);
    cfg.blockDim = dim3(kDx3Threads);
    cfg.dynamicSmemBytes = pr.pl.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    int na = 0;
    static const int no_pdl = env_int("DCG_TC_NO_PDL");
    if (!no_pdl) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    const cudaError_t err = five
                                ? cudaLaunchKernelEx(&cfg, conv_dx3_kernel<5, 5>, pr.ma, pr.mb, p, pr.dx3_args)
                                : cudaLaunchKernelEx(&cfg, conv_dx3_kernel<0, 0>, pr.ma, pr.mb, p, pr.dx3_args);
    if (err != cudaSuccess) return fail(DCG_ERR_CUDA, "conv_dx3_kernel launch: %s", cudaGetErrorString(err));
    count_launch();
    return DCG_OK;
}

int launch_rgb(Prepared& pr, const float* x, float* out, const EpilogueArgs& ep, cudaStream_t stream)
{
    Params& p = pr.pl.p;
    using Kernel = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, Params, RgbArgs, const float*);
    static const Kernel kernels[2][2] = {{conv_fwd_rgb_kernel<16, false>, conv_fwd_rgb_kernel<16, true>},
                                         {conv_fwd_rgb_kernel<32, false>, conv_fwd_rgb_kernel<32, true>}};
    const int wide = pr.rgb_args.kwc > 16, even = p.sw * p.C % 2 == 0;
    static OncePerDevice once[2][2];
    DCG_CUDA(allow_smem(once[wide][even], kernels[wide][even], kMaxSmem));
    p.out = out;
    p.ep = ep;
    p.scratch = nullptr;
    p.skip_stage = g_test_skip_stage.load();
    p.wait_cycles = g_wait_cycles.load();
    // the results of the chain leave as bulk copies in no order: of results for the same tensor only the last one
    if (p.ep.pre_act == out) p.ep.pre_act = nullptr;
    if (p.ep.raw_out == out || (p.ep.raw_out && p.ep.raw_out == p.ep.pre_act)) p.ep.raw_out = nullptr;
    launch_pdl(kernels[wide][even], (unsigned)pr.pl.grid, kRgbThreads, pr.pl.smem, stream, pr.mb, pr.rgb_maps.map[0], pr.rgb_maps.map[1], pr.rgb_maps.map[2],
               pr.rgb_maps.map[3], pr.ma, p, pr.rgb_args, x);
    DCG_LAUNCH_CHECK("conv_fwd_rgb_kernel");
    return DCG_OK;
}

struct CacheKey {
    int dev, kind, x3;
    dcg_conv_desc d;
    const void *a, *b, *ws;
    size_t ws_bytes;
};

struct CacheEntry {
    CacheKey key;
    Prepared prep;
};

constexpr size_t kCacheEntries = 512;
std::mutex g_cache_mutex;
std::vector<CacheEntry> g_cache;
std::unordered_map<CacheKey, size_t, BytesHash<CacheKey>, BytesEqual<CacheKey>> g_cache_at;   // where in g_cache
size_t g_cache_next = 0;

// FWD: plan and maps for y = conv(x, k).  xp / k4 of a narrow-channel layer live in the scratch.
int build_fwd(const dcg_conv_desc& d, const float* x, const float* k, void* ws, size_t ws_bytes, Prepared& pr)
{
    Plan& pl = pr.pl;
    pr.rgb = plan_rgb(d, pl, pr.rgb_args);
    if (pr.rgb) {   // k [kh][kw * C + c][o] as (o%32, kw * C + c, kh, o/32), box (32, places, 32 / places, o/32), zero-filled beyond
        const cuuint64_t kwc = (cuuint64_t)pr.rgb_args.kwc, places = kwc <= 16 ? 16 : 32;
        const cuuint64_t dims[4] = {32, kwc, (cuuint64_t)d.kh, (cuuint64_t)(d.o / 32)};
        const cuuint64_t strides[3] = {(cuuint64_t)d.o * 4, kwc * d.o * 4, 128};
        const cuuint32_t box[4] = {32, (cuuint32_t)places, (cuuint32_t)(32 / places), (cuuint32_t)(d.o / 32)};
        const cuuint32_t es[4] = {1, 1, 1, 1};
        const int st = encode_map(&pr.mb, k, 4, dims, true, strides, box, es);
        if (st || !pr.rgb_args.tma) return st;
        const cuuint64_t line = (cuuint64_t)d.w * d.c;   // x as (w * c, h, n), plain rows
        const cuuint64_t xdims[3] = {line, (cuuint64_t)d.h, (cuuint64_t)d.n};
        const cuuint64_t xstrides[2] = {line * 4, line * d.h * 4};
        const cuuint32_t xbox[3] = {(cuuint32_t)pr.rgb_args.pitch, (cuuint32_t)(pr.rgb_args.rows / pl.p.TN), (cuuint32_t)pl.p.TN};
        return encode_map(&pr.ma, x, 3, xdims, CU_TENSOR_MAP_SWIZZLE_NONE, xstrides, xbox, es);
    }
    pl = Plan{};
    if (!plan_fwd(d, pl)) return fail(DCG_ERR_UNSUPPORTED, "conv fwd: shape not supported by the tensor path");
    const Params& p = pl.p;
    int st;
    if (p.narrow) {
        if (!ws || ws_bytes < pl.ws_bytes)
            return fail(DCG_ERR_WORKSPACE, "conv (tensor path, narrow input): workspace %zu < %zu bytes", ws_bytes, pl.ws_bytes);
        uint8_t* base = static_cast<uint8_t*>(ws);
        const float* xp = reinterpret_cast<const float*>(base + pl.xp_off());
        const float* k4 = reinterpret_cast<const float*>(base + pl.k4_off());
        if ((st = map_window(&pr.ma, xp, d, pl, p.TW, p.TH, p.TN, false, 1))) return st;
        // k4 [kh][slot][o] as (o%32, slot, kh, o/32), box (32, 32, 1, bn/32)
        const cuuint64_t dims[4] = {32, 32, (cuuint64_t)d.kh, (cuuint64_t)(pad32(d.o) / 32)};
        const cuuint64_t strides[3] = {(cuuint64_t)pad32(d.o) * 4, (cuuint64_t)32 * pad32(d.o) * 4, 128};
        const cuuint32_t box[4] = {32, 32, 1, (cuuint32_t)(p.bn / 32)};
        const cuuint32_t es[4] = {1, 1, 1, 1};
        return encode_map(&pr.mb, k4, 4, dims, true, strides, box, es);
    }
    if ((st = map_act_4d(&pr.ma, x, d.n, d.h, d.w, d.c, p.TW, p.TH, p.TN, d.stride_w, d.stride_h))) return st;
    if (p.mt == 0) {   // k [tap][c][o] as (o, c, tap, 1), box (32, 32, 1, 1)
        const cuuint64_t dims[4] = {(cuuint64_t)d.o, (cuuint64_t)d.c, (cuuint64_t)(d.kh * d.kw), 1};
        const cuuint64_t strides[3] = {(cuuint64_t)d.o * 4, (cuuint64_t)d.c * d.o * 4, (cuuint64_t)d.kh * d.kw * d.c * d.o * 4};
        const cuuint32_t box[4] = {32, 32, 1, 1};
        const cuuint32_t es[4] = {1, 1, 1, 1};
        return encode_map(&pr.mb, k, 4, dims, true, strides, box, es);
    }
    // k [tap][c][o] as (o%32, c, tap, o/32), box (32, 32, 1, bn/32)
    const cuuint64_t dims[4] = {32, (cuuint64_t)d.c, (cuuint64_t)(d.kh * d.kw), (cuuint64_t)(d.o / 32)};
    const cuuint64_t strides[3] = {(cuuint64_t)d.o * 4, (cuuint64_t)d.c * d.o * 4, 128};
    const cuuint32_t box[4] = {32, 32, 1, (cuuint32_t)(p.bn / 32)};
    const cuuint32_t es[4] = {1, 1, 1, 1};
    return encode_map(&pr.mb, k, 4, dims, true, strides, box, es);
}

int build_dx(const dcg_conv_desc& d, const float* dy, const float* k, void* ws, size_t ws_bytes, Prepared& pr)
{
    Plan& pl = pr.pl;
    pr.dx3 = plan_dx3(d, pl, pr.dx3_args);
    if (pr.dx3) {
        // dy [n, ho, wo, o] in boxes of (32 o, 32 pixels, 4 rows, 1 image); k [tap][c][o] as (o, c, tap) in boxes of
        // (32 o, 4 c, 32 taps): rows 4 * tap + c, K-major, channel 3 and the taps beyond the last zero-filled
        int st = map_act_4d(&pr.ma, dy, d.n, d.ho, d.wo, d.o, 32, 4, 1, 1, 1);
        if (st) return st;
        const cuuint64_t dims[3] = {(cuuint64_t)d.o, (cuuint64_t)d.c, (cuuint64_t)(d.kh * d.kw)};
        const cuuint64_t strides[2] = {(cuuint64_t)d.o * 4, (cuuint64_t)d.c * d.o * 4};
        const cuuint32_t box[3] = {32, 4, 32};
        const cuuint32_t es[3] = {1, 1, 1};
        return encode_map(&pr.mb, k, 3, dims, false, strides, box, es);
    }
    pl = Plan{};
    pr.dxf = plan_dxf(d, pl, pr.cf);
    if (!pr.dxf) {
        pl = Plan{};
        if (!plan_dx(d, pl)) return fail(DCG_ERR_UNSUPPORTED, "conv dx: shape not supported by the tensor path");
    }
    const Params& p = pl.p;
    int st = map_act_4d(&pr.ma, dy, d.n, d.ho, d.wo, d.o, p.TW, p.TH, p.TN, 1, 1);
    if (st) return st;
    if (pl.ycol_bytes) {   // narrow-channel layer: GEMM over all taps, then gather
        if (!ws || ws_bytes < pl.ws_bytes)
            return fail(DCG_ERR_WORKSPACE, "conv dx (tensor path, narrow input): workspace %zu < %zu bytes", ws_bytes, pl.ws_bytes);
        if (short_ok(pl) && d.c <= 4 && d.kh * d.kw <= 32 && p.bn == 128) {
            // persistent GEMM: B straight from k [tap][c][o] as (o, c, tap) with a (32 o, 4 c, 32 taps) box - rows
            // 4 * tap + c of 32 contiguous o, K-major; channel 3 and the taps beyond the last are zero-filled
            pl.p.b_direct = 1;
            const cuuint64_t dims[3] = {(cuuint64_t)d.o, (cuuint64_t)d.c, (cuuint64_t)(d.kh * d.kw)};
            const cuuint64_t strides[2] = {(cuuint64_t)d.o * 4, (cuuint64_t)d.c * d.o * 4};
            const cuuint32_t box[3] = {32, 4, 32};
            const cuuint32_t es[3] = {1, 1, 1};
            return encode_map(&pr.mb, k, 3, dims, false, strides, box, es);
        }
        const float* k2 = reinterpret_cast<const float*>(static_cast<uint8_t*>(ws) + pl.k2_off());
        const int Jp = pl.Jp;
        // k2 [o][Jp] as (j%32, o, 1, j/32), box (32, 32, 1, bn/32): the FWD kernel's weight view with one tap
        const cuuint64_t dims[4] = {32, (cuuint64_t)d.o, 1, (cuuint64_t)(Jp / 32)};
        const cuuint64_t strides[3] = {(cuuint64_t)Jp * 4, (cuuint64_t)d.o * Jp * 4, 128};
        const cuuint32_t box[4] = {32, 32, 1, (cuuint32_t)(p.bn / 32)};
        const cuuint32_t es[4] = {1, 1, 1, 1};
        return encode_map(&pr.mb, k2, 4, dims, true, strides, box, es);
    }
    // k [kh][kw][c][o] as (o, c, kw, kh), box (32 o, bn c, 1, 1)
    const cuuint64_t dims[4] = {(cuuint64_t)d.o, (cuuint64_t)d.c, (cuuint64_t)d.kw, (cuuint64_t)d.kh};
    const cuuint64_t strides[3] = {(cuuint64_t)d.o * 4, (cuuint64_t)d.c * d.o * 4, (cuuint64_t)d.kw * d.c * d.o * 4};
    const cuuint32_t box[4] = {32, (cuuint32_t)p.bn, 1, 1};
    const cuuint32_t es[4] = {1, 1, 1, 1};
    return encode_map(&pr.mb, k, 4, dims, false, strides, box, es);
}

// DK: ma / mb are the maps of the A / B operand (x and dy, or dy and x when the roles are swapped).
int build_dk(const dcg_conv_desc& d, const float* x, const float* dy, void* ws, size_t ws_bytes, Prepared& pr)
{
    Plan& pl = pr.pl;
    if (!plan_dk(d, pl, ws ? ws_bytes : 0)) return fail(DCG_ERR_UNSUPPORTED, "conv dk: shape not supported by the tensor path");
    const Params& p = pl.p;
    CUtensorMap mx, mdy;
    int st;
    if (p.narrow) {
        if (!ws || ws_bytes < pl.ws_bytes)
            return fail(DCG_ERR_WORKSPACE, "conv (tensor path, narrow input): workspace %zu < %zu bytes", ws_bytes, pl.ws_bytes);
        const float* xp = reinterpret_cast<const float*>(static_cast<uint8_t*>(ws) + pl.xp_off());
        if ((st = map_window(&mx, xp, d, pl, p.TW, p.TH, p.TN, true, p.bn / 32))) return st;
        st = p.mt == 0 ? map_act_4d(&mdy, dy, d.n, d.ho, d.wo, d.o, p.TW, p.TH, p.TN, 1, 1, true)
                       : map_act_5d(&mdy, dy, d.n, d.ho, d.wo, d.o, p.TW, p.TH, p.TN, 1, 1, BM / 32);
        if (st) return st;
        pr.ma = mdy; pr.mb = mx;
        return DCG_OK;
    }
    if (p.mt == 0) {
        if ((st = map_act_4d(&mx, x, d.n, d.h, d.w, d.c, p.TW, p.TH, p.TN, d.stride_w, d.stride_h, true))) return st;
        if ((st = map_act_4d(&mdy, dy, d.n, d.ho, d.wo, d.o, p.TW, p.TH, p.TN, 1, 1, true))) return st;
        pr.ma = p.swap ? mdy : mx;
        pr.mb = p.swap ? mx : mdy;
        return DCG_OK;
    }
    const int x_chunks = p.swap ? p.bn / 32 : BM / 32 / p.mt, dy_chunks = p.swap ? BM / 32 : p.bn / 32;
    if ((st = map_act_5d(&mx, x, d.n, d.h, d.w, d.c, p.TW, p.TH, p.TN, d.stride_w, d.stride_h, x_chunks))) return st;
    if ((st = map_act_5d(&mdy, dy, d.n, d.ho, d.wo, d.o, p.TW, p.TH, p.TN, 1, 1, dy_chunks))) return st;
    if (p.swap) { pr.ma = mdy; pr.mb = mx; }
    else { pr.ma = mx; pr.mb = mdy; }
    return DCG_OK;
}

// Looks the call up, building and filing it on a miss.  The entry is copied out under the lock.
int prepared_call(int kind, const dcg_conv_desc& d, const void* a, const void* b, void* ws, size_t ws_bytes, Prepared& out, CacheKey& key)
{
    std::memset(&key, 0, sizeof(key));
    if (cudaGetDevice(&key.dev) != cudaSuccess) key.dev = -1;
    key.kind = kind; key.x3 = t_plan_x3 | (dxf_mode() << 1);   // the plan depends on both
    key.d = d; key.a = a; key.b = b; key.ws = ws; key.ws_bytes = ws_bytes;
    {
        std::lock_guard<std::mutex> lock(g_cache_mutex);
        const auto it = g_cache_at.find(key);
        if (it != g_cache_at.end()) { out = g_cache[it->second].prep; return DCG_OK; }
    }
    int st;
    switch (kind) {
    case kConvFwd: st = build_fwd(d, static_cast<const float*>(a), static_cast<const float*>(b), ws, ws_bytes, out); break;
    case kConvDx: st = build_dx(d, static_cast<const float*>(a), static_cast<const float*>(b), ws, ws_bytes, out); break;
    default: st = build_dk(d, static_cast<const float*>(a), static_cast<const float*>(b), ws, ws_bytes, out); break;
    }
    if (st) return st;
    std::lock_guard<std::mutex> lock(g_cache_mutex);
    if (g_cache_at.count(key)) return DCG_OK;   // another thread was faster
    if (g_cache.size() < kCacheEntries) {
        g_cache_at[key] = g_cache.size();
        g_cache.push_back(CacheEntry{key, out});
    } else {
        g_cache_at.erase(g_cache[g_cache_next].key);
        g_cache_at[key] = g_cache_next;
        g_cache[g_cache_next] = CacheEntry{key, out};
        g_cache_next = (g_cache_next + 1) % kCacheEntries;
    }
    return DCG_OK;
}

// Brings the output-side maps of an RGB forward in line with this call's tensors (boxes of 32 pixels x 32 channels, the rows of an
// epilogue warp) and files those that were not there.
int rgb_maps(const dcg_conv_desc& d, const CacheKey& key, const void* const (&tensors)[4], Prepared& pr)
{
    const Params& p = pr.pl.p;
    const int tw = std::min(p.TW, 32), th = std::min(p.TH, 32 / tw), tn = 32 / (tw * th);
    RgbMaps& m = pr.rgb_maps;
    bool fresh = false;
    for (int i = 0; i < 4; ++i) {
        if (!tensors[i] || tensors[i] == m.of[i]) continue;   // (absent ones are not read)
        const int st = map_act_4d(&m.map[i], static_cast<const float*>(tensors[i]), d.n, d.ho, d.wo, d.o, tw, th, tn, 1, 1);
        if (st) return st;
        m.of[i] = tensors[i];
        fresh = true;
    }
    if (!fresh) return DCG_OK;
    std::lock_guard<std::mutex> lock(g_cache_mutex);
    const auto it = g_cache_at.find(key);
    if (it != g_cache_at.end()) g_cache[it->second].prep.rgb_maps = m;
    return DCG_OK;
}

// ---- what the entry points ask before a call: does the tensor path take the shape, and how much scratch does it need ----
struct QueryAnswer {
    bool supported;
    size_t ws_bytes, ws_least;   // what the best plan takes, and what the call can do with
};
std::mutex g_query_mutex;
std::unordered_map<QueryKey, QueryAnswer, BytesHash<QueryKey>, BytesEqual<QueryKey>> g_query;

QueryAnswer query(const dcg_conv_desc& d, int kind, bool x3)
{
    const QueryKey key = query_key(d, kind, x3);
    {
        std::lock_guard<std::mutex> lock(g_query_mutex);
        const auto it = g_query.find(key);
        if (it != g_query.end()) return it->second;
    }
    PlanX3 scope(x3);
    Plan pl;
    QueryAnswer a{make_plan(d, kind, pl), 0, 0};
    if (a.supported) a.ws_bytes = a.ws_least = pl.ws_bytes;
    Plan least;
    if (a.supported && kind == kConvDk && make_plan(d, kind, least, 0)) a.ws_least = least.ws_bytes;
    std::lock_guard<std::mutex> lock(g_query_mutex);
    if (g_query.size() >= 4096) g_query.clear();
    g_query[key] = a;
    return a;
}

}  // namespace

bool conv_tc_supported(const dcg_conv_desc& d, int kind, bool x3) { return query(d, kind, x3).supported; }

size_t conv_tc_workspace(const dcg_conv_desc& d, int kind, bool x3) { return query(d, kind, x3).ws_bytes; }
size_t conv_tc_workspace_least(const dcg_conv_desc& d, int kind, bool x3) { return query(d, kind, x3).ws_least; }

int conv_tc_fwd(const dcg_conv_desc& d, const float* x, const float* k, float* y, const EpilogueArgs& ep,
                void* ws, size_t ws_bytes, cudaStream_t stream, bool x3)
{
    PlanX3 scope(x3);
    Prepared pr;
    CacheKey key;
    int st = prepared_call(kConvFwd, d, x, k, ws, ws_bytes, pr, key);
    if (st) return st;
    if (pr.rgb) {
        const void* const tensors[4] = {y, ep.raw_out, ep.pre_act, ep.gate};
        if ((st = rgb_maps(d, key, tensors, pr))) return st;
        return launch_rgb(pr, x, y, ep, stream);
    }
    if (pr.pl.p.narrow) {
        float *xp, *k4;
        if ((st = narrow_prepare(d, pr.pl, x, k, ws, ws_bytes, stream, &xp, &k4))) return st;
        if (short_ok(pr.pl)) return launch_short(pr, true, y, ep, stream);
    }
    return launch<MODE_FWD>(pr.ma, pr.mb, pr.pl, y, ep, d.o, ws, ws_bytes, stream);
}

int conv_tc_dx(const dcg_conv_desc& d, const float* dy, const float* k, float* dx, const EpilogueArgs& ep,
               void* ws, size_t ws_bytes, cudaStream_t stream, bool x3)
{
    PlanX3 scope(x3);
    Prepared pr;
    CacheKey key;
    int st = prepared_call(kConvDx, d, dy, k, ws, ws_bytes, pr, key);
    if (st) return st;
    Plan& pl = pr.pl;
    if (pr.dx3) return launch_dx3(pr, dx, ep, stream);
    if (pl.ycol_bytes) {   // narrow-channel layer: GEMM over all taps, then gather
        uint8_t* base = static_cast<uint8_t*>(ws);
        float* k2 = reinterpret_cast<float*>(base + pl.k2_off());
        float* ycol = reinterpret_cast<float*>(base + pl.ycol_off());
        const int Jp = pl.Jp;
        if (!pl.p.b_direct) {   // the transposed weights k2 [o][Jp]; the persistent GEMM reads k itself
            launch_pdl(repack_k2_kernel, (d.o * Jp + 255) / 256, 256, 0, stream, k, k2, d.kh * d.kw, d.c, Jp, d.o);
            DCG_LAUNCH_CHECK("repack_k2_kernel");
        }
        const EpilogueArgs none{};
        if (short_ok(pl)) st = launch_short(pr, false, ycol, none, stream);
        else st = launch<MODE_FWD>(pr.ma, pr.mb, pl, ycol, none, Jp, ws, ws_bytes, stream);
        if (st) return st;
        const size_t total = (size_t)d.n * d.h * d.w;
        size_t blocks = (total + 255) / 256;
        const size_t cap = (size_t)sm_count() * 16;
        if (blocks > cap) blocks = cap;
        if (d.kh == 5 && d.kw == 5 && d.stride_h == 2 && d.stride_w == 2)
            launch_pdl(col2im_kernel<5, 5, 2>, (unsigned)blocks, 256, 0, stream, reinterpret_cast<const float4*>(ycol), dx, d.n, d.h,
                       d.w, d.c, d.ho, d.wo, d.kh, d.kw, d.stride_h, d.stride_w, d.pad_top, d.pad_left, ep);
        else
            launch_pdl(col2im_kernel<0, 0, 0>, (unsigned)blocks, 256, 0, stream, reinterpret_cast<const float4*>(ycol), dx, d.n, d.h,
                       d.w, d.c, d.ho, d.wo, d.kh, d.kw, d.stride_h, d.stride_w, d.pad_top, d.pad_left, ep);
        DCG_LAUNCH_CHECK("col2im_kernel");
        return DCG_OK;
    }
    if (pr.dxf) return launch_dxf(pr, dx, ep, stream);
    return launch<MODE_DX>(pr.ma, pr.mb, pl, dx, ep, d.c, ws, ws_bytes, stream);
}

int conv_tc_dk(const dcg_conv_desc& d, const float* x, const float* dy, float* dk, void* ws, size_t ws_bytes,
               cudaStream_t stream, bool x3)
{
    PlanX3 scope(x3);
    Prepared pr;
    CacheKey key;
    int st = prepared_call(kConvDk, d, x, dy, ws, ws_bytes, pr, key);
    if (st) return st;
    if (pr.pl.p.narrow) {
        float* xp;
        if ((st = narrow_prepare(d, pr.pl, x, nullptr, ws, ws_bytes, stream, &xp, nullptr))) return st;
    }
    const EpilogueArgs none{};
    return launch<MODE_DK>(pr.ma, pr.mb, pr.pl, dk, none, d.o, ws, ws_bytes, stream);
}

bool conv_tc_plan(const dcg_conv_desc& d, int kind, bool x3, int plan[6])
{
    PlanX3 scope(x3);
    Plan pl;
    RgbArgs rgb;
    const bool is_rgb = kind == kConvFwd && plan_rgb(d, pl, rgb);
    if (!is_rgb) {
        pl = Plan{};
        if (!make_plan(d, kind, pl)) return false;
    }
    const Params& p = pl.p;
    // what the kernel allocates: two accumulators in a power of two of columns where it is persistent
    int tmem = tmem_columns(p.kind, p.bn, p.x3_slots);
    if (p.walk || is_rgb)
        for (tmem = 32; tmem < 2 * p.bn;) tmem <<= 1;
    const int values[6] = {p.bn, p.n_tiles, p.splits, p.stages, tmem, (int)pl.smem};
    for (int i = 0; i < 6; ++i) plan[i] = values[i];
    return true;
}

bool conv_tc_form(const dcg_conv_desc& d, int kind, bool x3, int form[4])
{
    PlanX3 scope(x3);
    Prepared pr;
    Plan& pl = pr.pl;
    int kernel = DCG_FORM_TILES;
    if (kind == kConvFwd && plan_rgb(d, pl, pr.rgb_args)) kernel = DCG_FORM_RGB;
    else if (kind == kConvDx && plan_dx3(d, pl, pr.dx3_args)) kernel = DCG_FORM_RGB_GRAD;
    else if (kind == kConvDx && plan_dxf(d, pl = Plan{}, pr.cf)) kernel = DCG_FORM_CLASSES;
    else {
        pl = Plan{};
        if (!make_plan(d, kind, pl)) return false;
        if (pl.p.walk) kernel = DCG_FORM_WALK;
        else if ((pl.p.narrow || pl.ycol_bytes) && kind != kConvDk && short_ok(pl)) kernel = DCG_FORM_SHORT;
    }
    const Params& p = pl.p;
    form[0] = kernel;
    form[1] = p.ext_finish;
    form[2] = kernel == DCG_FORM_TILES ? epilogue_groups(p.kind) : 0;
    form[3] = kernel == DCG_FORM_TILES && p.x3 ? p.x3_slots : 0;
    return true;
}

void conv_tc_set_dx_mode(int mode) { g_dxf_mode.store(mode < 0 || mode > 2 ? -1 : mode); }
unsigned long long conv_tc_fused_dx_launches() { return g_dxf_launches.load(); }
unsigned long long conv_tc_dx_plans() { return g_dx_plans.load(); }
unsigned long long conv_tc_maps_encoded() { return g_maps_encoded.load(); }

// wait_cycles: > 0 sets the limit, -1 restores the default, 0 leaves it; skip_stage: -2 leaves it.
void conv_tc_set_hooks(long long wait_cycles, int skip_stage)
{
    if (wait_cycles > 0) g_wait_cycles.store(wait_cycles);
    else if (wait_cycles < 0) g_wait_cycles.store(default_wait_cycles());
    if (skip_stage != -2) g_test_skip_stage.store(skip_stage);
}

// Reads (and clears) the device status word of the tensor-path kernels.  Synchronises the device.
int conv_tc_device_status(int* detail /* [4] */)
{
    int h[4] = {0, 0, 0, 0};
    DCG_CUDA(cudaDeviceSynchronize());
    DCG_CUDA(cudaMemcpyFromSymbol(h, g_tc_status, sizeof(h)));
    if (detail) for (int i = 0; i < 4; ++i) detail[i] = h[i];
    if (h[0] != 0) {
        const int zero[4] = {0, 0, 0, 0};
        DCG_CUDA(cudaMemcpyToSymbol(g_tc_status, zero, sizeof(zero)));
        return fail(DCG_ERR_DEVICE, "tensor-path kernel gave up waiting: code %d block %d role %d stage %d",
                    h[0], h[1], h[2], h[3]);
    }
    return dp_status_check();
}

}  // namespace dcg

extern "C" int dcg_device_status(void) { return dcg::conv_tc_device_status(nullptr); }

extern "C" void dcg_debug_set_wait_limit(long long sm_clocks)
{
    dcg::conv_tc_set_hooks(sm_clocks > 0 ? sm_clocks : -1, -2);
}

extern "C" void dcg_debug_skip_stage(int stage) { dcg::conv_tc_set_hooks(0, stage < 0 ? -1 : stage); }

extern "C" void dcg_debug_set_dx_mode(int mode) { dcg::conv_tc_set_dx_mode(mode); }
extern "C" int dcg_debug_conv_plan(const dcg_conv_desc* desc, int kind, int precision, int plan[6])
{
    const int st = dcg::conv_check_desc(desc, "dcg_debug_conv_plan");
    if (st) return st;
    if (precision == DCG_PREC_FP32 || !plan || !dcg::conv_tc_plan(*desc, kind, precision == DCG_PREC_3XTF32, plan)) return DCG_ERR_UNSUPPORTED;
    return DCG_OK;
}

extern "C" int dcg_debug_conv_form(const dcg_conv_desc* desc, int kind, int precision, int form[4])
{
    const int st = dcg::conv_check_desc(desc, "dcg_debug_conv_form");
    if (st) return st;
    if (precision == DCG_PREC_FP32 || !form || !dcg::conv_tc_form(*desc, kind, precision == DCG_PREC_3XTF32, form)) return DCG_ERR_UNSUPPORTED;
    return DCG_OK;
}

extern "C" uint64_t dcg_debug_dx_plans(void) { return dcg::conv_tc_dx_plans(); }
extern "C" uint64_t dcg_debug_maps_encoded(void) { return dcg::conv_tc_maps_encoded(); }
extern "C" uint64_t dcg_debug_fused_dx_launches(void) { return dcg::conv_tc_fused_dx_launches(); }

#ifdef DCG_TC_TRACING
// Tuning aids of -DDCG_TC_TRACING builds, not part of the public header: copy the timelines recorded
// by the last tensor-path launch (DCG_TC_DEBUG bits 4 / 8) to `out`.  Synchronise the device.
extern "C" int dcg_debug_cta_trace(unsigned long long* out /* [1024][8] */)
{
    if (cudaDeviceSynchronize() != cudaSuccess) return DCG_ERR_CUDA;
    return cudaMemcpyFromSymbol(out, dcg::g_tc_cta_trace, sizeof(unsigned long long) * 1024 * 8) == cudaSuccess ? DCG_OK : DCG_ERR_CUDA;
}

extern "C" int dcg_debug_trace(long long* out /* [3080] */)
{
    if (cudaDeviceSynchronize() != cudaSuccess) return DCG_ERR_CUDA;
    return cudaMemcpyFromSymbol(out, dcg::g_tc_trace, sizeof(long long) * 3080) == cudaSuccess ? DCG_OK : DCG_ERR_CUDA;
}
#endif

// CUDA-core fp32 convolution kernels (DCG_PREC_FP32, and every shape the tensor path cannot take).
//
// They are written for exactness first: each output is accumulated in the order the reference's CPU code
// uses, with unfused IEEE multiplies and adds, so the results are bit-comparable with src/cpu/ops.hxx:
//   forward      : one accumulator over (channel, kernel row, kernel column), ops.hxx:227-246
//   input grad   : per output filter an inner sum over taps, filters added in order, ops.hxx:650-679
//   kernel grad  : per image an inner sum over output pixels, images added in order, ops.hxx:754-772
// Within that order there is no K split; what is free is how the outputs are spread over threads and how
// the operands reach them.  conv_ordered_fwd_kernel, conv_ordered_dx_kernel (by parity class) and
// conv_ordered_dk_kernel are register-tiled GEMMs on operand tiles that cp.async gathers straight from the
// NHWC / HWIO tensors; the conv_*_generic kernels further down (one thread per output, as
// src/gpu/conv2d_naive.hh) remain for kernels with more than kOrdMaxTaps taps, whose tiles would not fit.
#include <type_traits>

#include "common.cuh"
#include "conv.cuh"

namespace dcg {
namespace {

constexpr int kThreads = 128;

constexpr int kOrdSmem = 227 * 1024;
constexpr int kOrdMaxTaps = 25;   // taps of one accumulation chain: bounds the operand tiles in shared memory

__device__ __forceinline__ void cp_async4(uint32_t dst, const float* src, bool in)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(in ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const float* src, bool in)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// W consecutive floats of an operand tile
template <int W>
__device__ __forceinline__ void lds_vec(const float* s, float (&v)[W])
{
    if constexpr (W == 1) {
        v[0] = *s;
    } else if constexpr (W == 2) {
        const float2 t = *reinterpret_cast<const float2*>(s);
        v[0] = t.x; v[1] = t.y;
    } else {
        static_assert(W == 4, "1, 2 or 4 floats");
        const float4 t = *reinterpret_cast<const float4*>(s);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    }
}

// ---- one output as the reference's loops have it ------------------------------------------------------------
// y[pixel, o] of pixel number `pixel`
__device__ __forceinline__ float fwd_sum(const float* __restrict__ x, const float* __restrict__ k, const dcg_conv_desc& d, size_t pixel, int o)
{
    const int j = (int)(pixel % d.wo);
    size_t t = pixel / d.wo;
    const int i = (int)(t % d.ho);
    const int n = (int)(t / d.ho);
    const int h0 = i * d.stride_h - d.pad_top, w0 = j * d.stride_w - d.pad_left;
    const float* xn = x + (size_t)n * d.h * d.w * d.c;
    float val = 0.f;
    for (int q = 0; q < d.c; ++q)
        for (int di = 0; di < d.kh; ++di) {
            const int h = h0 + di;
            if (h < 0 || h >= d.h) continue;
            for (int dj = 0; dj < d.kw; ++dj) {
                const int w = w0 + dj;
                if (w < 0 || w >= d.w) continue;
                const float xv = __ldg(xn + ((size_t)h * d.w + w) * d.c + q);
                const float kv = __ldg(k + (((size_t)di * d.kw + dj) * d.c + q) * d.o + o);
                val = __fadd_rn(val, __fmul_rn(xv, kv));
            }
        }
    return val;
}

// dx[n,i,j,c] = sum_o ( sum_{di,dj} dyz[n,i+di-P,j+dj-Q,o] * k[KH-1-di,KW-1-dj,c,o] ), dyz the
// zero-inserted dy, P = KH-1-pad_top, Q = KW-1-pad_left (src/cpu/ops.hxx:618-629).
__device__ __forceinline__ float dx_sum(const float* __restrict__ dy, const float* __restrict__ k, const dcg_conv_desc& d, size_t pixel, int c)
{
    const int j = (int)(pixel % d.w);
    size_t t = pixel / d.w;
    const int i = (int)(t % d.h);
    const int n = (int)(t / d.h);
    const int P = d.kh - 1 - d.pad_top, Q = d.kw - 1 - d.pad_left;
    const float* dyn = dy + (size_t)n * d.ho * d.wo * d.o;
    float total_v = 0.f;
    for (int o = 0; o < d.o; ++o) {
        float val = 0.f;
        for (int di = 0; di < d.kh; ++di) {
            const int ph = i + di - P;
            if (ph < 0 || ph % d.stride_h != 0) continue;
            const int a = ph / d.stride_h;
            if (a >= d.ho) continue;
            for (int dj = 0; dj < d.kw; ++dj) {
                const int pw = j + dj - Q;
                if (pw < 0 || pw % d.stride_w != 0) continue;
                const int b = pw / d.stride_w;
                if (b >= d.wo) continue;
                const float g = __ldg(dyn + ((size_t)a * d.wo + b) * d.o + o);
                const float kv = __ldg(k + (((size_t)(d.kh - 1 - di) * d.kw + (d.kw - 1 - dj)) * d.c + c) * d.o + o);
                val = __fadd_rn(val, __fmul_rn(g, kv));
            }
        }
        total_v = (o == 0) ? val : __fadd_rn(total_v, val);
    }
    return total_v;
}

// dk[row, o] = sum_n ( sum_{a,b} x[n,kh+s*a-pt,kw+s*b-pl,c] * dy[n,a,b,o] ), row = (kh * KW + kw) * C + c
__device__ __forceinline__ float dk_sum(const float* __restrict__ x, const float* __restrict__ dy, const dcg_conv_desc& d, size_t row, int o)
{
    const int c = (int)(row % d.c);
    size_t t = row / d.c;
    const int kw = (int)(t % d.kw);
    const int kh = (int)(t / d.kw);
    float total_v = 0.f;
    for (int n = 0; n < d.n; ++n) {
        const float* xn = x + (size_t)n * d.h * d.w * d.c;
        const float* dyn = dy + (size_t)n * d.ho * d.wo * d.o;
        float val = 0.f;
        for (int a = 0; a < d.ho; ++a) {
            const int h = kh + d.stride_h * a - d.pad_top;
            if (h < 0 || h >= d.h) continue;
            for (int b = 0; b < d.wo; ++b) {
                const int w = kw + d.stride_w * b - d.pad_left;
                if (w < 0 || w >= d.w) continue;
                const float xv = __ldg(xn + ((size_t)h * d.w + w) * d.c + c);
                const float g = __ldg(dyn + ((size_t)a * d.wo + b) * d.o + o);
                val = __fadd_rn(val, __fmul_rn(xv, g));
            }
        }
        total_v = (n == 0) ? val : __fadd_rn(total_v, val);
    }
    return total_v;
}

// The ordered kernels multiply taps outside the image as zeros where the reference skips them.  That adds +0 and leaves the same
// bits unless the other factor is infinite or NaN: then the result is NaN.  They note in g_nan_seen that there is one - for good,
// so that launches of several streams need no order - and conv_nan_again_kernel behind them, which ends at once as long as there
// has been none, computes NaN outputs again with the sums above.  (Sums in the ordered kernels themselves, called or inlined,
// take registers from the main loops: training step at batch 8 6.11 -> 6.25 to 6.46 ms.  The launch between them is 0.3 to 0.9 us
// of a layer by itself; in a list it also keeps the long blocks of the next kernel from starting early and piling up on the SMs
// that are free first, 5.25 ms.)  The kernels of small input and kernel gradients, for which a launch is long, do have such sums,
// with 32-bit indexes and nothing unrolled; theirs cost nothing (9 x 9 x 5 images, 5 x 5: input gradient 4.5 us, 5.2 with a launch).
__host__ __device__ constexpr bool dx_again_inside(int tm) { return tm == 1; }
__host__ __device__ constexpr bool dk_again_inside(int tm, int tn) { return tm * tn <= 4; }
__device__ int g_nan_seen;
template <int TM, int TN>
__device__ __forceinline__ bool any_nan(const float (&v)[TM][TN])
{
    bool nan = false;
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) nan = nan || isnan(v[i][j]);
    return nan;
}

enum OrderedKind { kOrdFwd, kOrdDx, kOrdDk };
template <int KIND>
__global__ void __launch_bounds__(kThreads)
conv_nan_again_kernel(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ out, const dcg_conv_desc d, const EpilogueArgs ep,
                      const size_t total)
{
    pdl_enter();
    if (*reinterpret_cast<volatile int*>(&g_nan_seen) == 0) return;
    const int cols = KIND == kOrdDx ? d.c : d.o;
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
        if (!isnan(out[idx])) continue;
        const size_t row = idx / cols;
        const int col = (int)(idx % cols);
        if (KIND == kOrdFwd) out[idx] = epilogue_apply(ep, fwd_sum(a, b, d, row, col), idx, col);
        else if (KIND == kOrdDx) out[idx] = epilogue_apply(ep, dx_sum(a, b, d, row, col), idx, col);
        else out[idx] = dk_sum(a, b, d, row, col);
    }
}

// ---- forward and input gradient as ordered implicit GEMMs -----------------------------------------------
// out[pixel, channel] over K = (contracted channel q outermost, tap innermost), the reference's loop nest.
// An operand whose contracted channel is its contiguous axis (x, dy, and the weights of the input gradient) is
// gathered sixteen bytes - four channels of one (row, tap) - at a time with cp.async and kept as it comes:
// [row][channel quad][tap][4], row pitch 4 mod 8 words so that eight rows start in different bank quads.  The
// weights of the forward are rows of output channels, [q][tap][channel].  Taps outside the image are zero-filled
// (see g_nan_seen).  Two to four stages of QC channels x all taps.
// Bound by issue (the sum must stay unfused: two instructions per product; packed f32x2 arithmetic was measured
// and is no faster, its operands have to be duplicated) and, where the outputs are few, by the latency of the
// chain of dependent adds.  Measured, 5x5 / stride 2 layers: 18 TFLOP/s (a multiply and an add counted as two) of the
// 37 that 148 x 128 lanes issue where a 4 x 4 thread tile is used, 7-11 at batch 8; the 256 -> 512 forward of 8
// images takes 122 us, one thread per output took 2.5 ms; a training iteration at batch 8 6.2 ms against 89.7.
struct OrdGeom {      // one class of output pixels and what its taps read
    int mh, mw;       // pixels of the class
    int SH, SW, SC;   // the source tensor
    int Th, Tw;       // taps
    int eh, ew, sh, sw;   // source row of (pixel row i, tap row a): i * sh + eh + a
};

constexpr int kOrdQuads = 25;   // 16-byte words of one operand row in a stage: taps x channel quads, at most

// What one thread copies of a channel-contiguous operand tile in every stage: (row, quad, tap) items tid, tid + THREADS, ...
// Their places do not change from stage to stage - a stage only moves the channel on - so they are worked out once.
template <int ROWS, int THREADS>
struct Gather {
    static constexpr int ITEMS = (ROWS * kOrdQuads + THREADS - 1) / THREADS;
    int off[ITEMS];   // element offset of channel 0 of the item's quad, -1: zero-fill, -2: no item
    // src_off(row, tap): element offset of channel 0, or -1
    template <typename F>
    __device__ __forceinline__ void plan(int T, int quads, F src_off)
    {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const int idx = threadIdx.x + i * THREADS, row = idx % ROWS, tq = idx / ROWS;
            off[i] = -2;
            if (tq < T * quads) {
                const int g = tq / T, o = src_off(row, tq - g * T);
                off[i] = o < 0 ? -1 : o + 4 * g;
            }
        }
    }
    __device__ __forceinline__ void load(uint32_t dst, int pitch, int T, const float* src, int q0, int qc, int SC, bool vec) const
    {
        const bool tail = q0 + qc > SC;
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            if (off[i] == -2) continue;
            const int idx = threadIdx.x + i * THREADS, row = idx % ROWS, tq = idx / ROWS;
            const uint32_t d = dst + 4u * (uint32_t)(row * pitch + 4 * tq);
            const int left = tail ? SC - q0 - 4 * (tq / T) : 4;   // channels of this quad that exist
            const bool in = off[i] >= 0;
            const float* s = src + (in ? off[i] + q0 : 0);
            if (vec) {
                cp_async16(d, s, in && left > 0);
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u) cp_async4(d + 4u * u, s + u, in && u < left);
            }
        }
    }
};

// Pixel rows of the A operand.
template <int ROWS, int THREADS>
__device__ __forceinline__ void gather_pixels(Gather<ROWS, THREADS>& ga, const OrdGeom& g, int quads, long long m0, long long pixels)
{
    ga.plan(g.Th * g.Tw, quads, [&](int row, int tap) {
        const long long p = m0 + row;
        if (p >= pixels) return -1;
        const int j = (int)(p % g.mw);
        const long long t = p / g.mw;
        const int a = tap / g.Tw, r = (int)(t % g.mh) * g.sh + g.eh + a, c = j * g.sw + g.ew + tap - a * g.Tw;
        if (r < 0 || r >= g.SH || c < 0 || c >= g.SW) return -1;
        return (int)((((t / g.mh) * g.SH + r) * g.SW + c) * g.SC);
    });
}

__host__ __device__ constexpr int ord_pitch(int tile) { return tile + 4; }
__host__ __device__ constexpr int ord_row_pitch(int taps, int qc) { return taps * qc % 8 == 0 ? taps * qc + 4 : taps * qc; }

template <int TM, int TN, int TX, int TY, int STAGES, int U>   // U divides the number of taps
__global__ void __launch_bounds__(TX * TY)
conv_ordered_fwd_kernel(const float* __restrict__ x, const float* __restrict__ k, float* __restrict__ y,
                        const dcg_conv_desc d, const EpilogueArgs ep, const int QC, const int vec_a, const int vec_b)
{
    constexpr int BMT = TM * TY, BNT = TN * TX, THREADS = TX * TY, LDB = ord_pitch(BNT);
    extern __shared__ __align__(16) float smem[];
    pdl_enter();
    const OrdGeom g{d.ho, d.wo, d.h, d.w, d.c, d.kh, d.kw, -d.pad_top, -d.pad_left, d.stride_h, d.stride_w};
    const int T = d.kh * d.kw, tid = threadIdx.x;
    const long long pixels = (long long)d.n * d.ho * d.wo, m0 = (long long)blockIdx.x * BMT;
    const int n0 = blockIdx.y * BNT;
    const int pitch = ord_row_pitch(T, QC), stage = BMT * pitch + QC * T * LDB;
    const uint32_t smem0 = (uint32_t)__cvta_generic_to_shared(smem);
    Gather<BMT, THREADS> ga;
    gather_pixels(ga, g, QC >> 2, m0, pixels);
    // weights: rows (q, tap) of output channels, sixteen bytes at a time where the channel count allows
    constexpr int COLS = BNT / 4, BITEMS = (4 * kOrdQuads * COLS + THREADS - 1) / THREADS;
    int boff[BITEMS];
#pragma unroll
    for (int i = 0; i < BITEMS; ++i) {
        const int idx = tid + i * THREADS, nn = 4 * (idx % COLS), r = idx / COLS, q = r / T;
        boff[i] = r < QC * T && n0 + nn < d.o ? ((r - q * T) * d.c + q) * d.o + n0 + nn : -1;
    }
    auto load_stage = [&](int q0, int buf) {
        const uint32_t as = smem0 + 4u * (uint32_t)(buf * stage), bs = as + 4u * (uint32_t)(BMT * pitch);
        ga.load(as, pitch, T, x, q0, QC, d.c, vec_a);
        if (vec_b) {
            const int rows = min(QC, d.c - q0) * T;
#pragma unroll
            for (int i = 0; i < BITEMS; ++i) {
                const int idx = tid + i * THREADS, r = idx / COLS;
                if (r < rows) cp_async16(bs + 4u * (uint32_t)(r * LDB + 4 * (idx % COLS)), k + (boff[i] < 0 ? 0 : boff[i] + q0 * d.o), boff[i] >= 0);
            }
        } else {
            for (int idx = tid; idx < min(QC, d.c - q0) * T * BNT; idx += THREADS) {
                const int nn = idx % BNT, r = idx / BNT, q = r / T;
                const bool in = n0 + nn < d.o;
                cp_async4(bs + 4u * (uint32_t)(r * LDB + nn), in ? k + ((long long)(r - q * T) * d.c + q0 + q) * d.o + n0 + nn : k, in);
            }
        }
        cp_async_commit();
    };

    const int tx = tid % TX, ty = tid / TX;
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s * QC < d.c) load_stage(s * QC, s);
        else cp_async_commit();
    }
    int buf = 0, next = STAGES - 1;
    for (int q0 = 0; q0 < d.c; q0 += QC) {
        if (q0 + (STAGES - 1) * QC < d.c) load_stage(q0 + (STAGES - 1) * QC, next);
        else cp_async_commit();
        next = next + 1 == STAGES ? 0 : next + 1;
        cp_async_wait<STAGES - 1>();
        __syncthreads();
        const float* as = smem + buf * stage + ty * pitch;
        const float* bs = smem + buf * stage + BMT * pitch + tx * TN;
        const int qn = min(QC, d.c - q0);
        for (int q = 0; q < qn; ++q) {
            const float* ap[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) ap[i] = as + i * TY * pitch + 4 * T * (q >> 2) + (q & 3);
            for (int t = 0; t < T; t += U, bs += U * LDB) {
                // operands and products of U taps first: only the adds form a chain
                float a[U][TM][1], b[U][TN];
#pragma unroll
                for (int u = 0; u < U; ++u) {
#pragma unroll
                    for (int i = 0; i < TM; ++i) lds_vec<1>(ap[i] + 4 * u, a[u][i]);
                    lds_vec<TN>(bs + u * LDB, b[u]);
                }
#pragma unroll
                for (int i = 0; i < TM; ++i) ap[i] += 4 * U;
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int i = 0; i < TM; ++i)
#pragma unroll
                        for (int j = 0; j < TN; ++j) acc[i][j] = __fadd_rn(acc[i][j], __fmul_rn(a[u][i][0], b[u][j]));
            }
        }
        __syncthreads();
        buf = buf + 1 == STAGES ? 0 : buf + 1;
    }
    if (any_nan(acc)) g_nan_seen = 1;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const long long p = m0 + ty + i * TY;
        if (p >= pixels) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int ch = n0 + tx * TN + j;
            if (ch >= d.o) continue;
            const size_t idx = (size_t)p * d.o + ch;
            y[idx] = epilogue_apply(ep, acc[i][j], idx, ch);
        }
    }
}

// Input gradient: the taps of one filter are summed first, the filters' sums added in order - so four filters at a time
// are four independent chains, read as 16-byte words of both operands.  Each parity class of output pixels
// (blockIdx.z) runs by itself: only taps that meet a dy pixel exist.
template <int TM, int TN, int TX, int TY, int STAGES>
__global__ void __launch_bounds__(TX * TY)
conv_ordered_dx_kernel(const float* __restrict__ dy, const float* __restrict__ k, float* __restrict__ dx,
                       const dcg_conv_desc d, const EpilogueArgs ep, const int QC, const int vec)
{
    constexpr int BMT = TM * TY, BNT = TN * TX, THREADS = TX * TY;
    extern __shared__ __align__(16) float smem[];
    pdl_enter();
    const int tid = threadIdx.x;
    const int P = d.kh - 1 - d.pad_top, Q = d.kw - 1 - d.pad_left;
    // first tap (in flipped order) of this class: in this order the classes with the most taps start first
    const int r0h = blockIdx.z / d.stride_w, r0w = blockIdx.z % d.stride_w;
    int ph = (P - r0h) % d.stride_h, pw = (Q - r0w) % d.stride_w;
    if (ph < 0) ph += d.stride_h;
    if (pw < 0) pw += d.stride_w;
    OrdGeom g;
    g.mh = (d.h - ph + d.stride_h - 1) / d.stride_h; g.mw = (d.w - pw + d.stride_w - 1) / d.stride_w;
    g.SH = d.ho; g.SW = d.wo; g.SC = d.o;
    g.Th = r0h < d.kh ? (d.kh - 1 - r0h) / d.stride_h + 1 : 0;
    g.Tw = r0w < d.kw ? (d.kw - 1 - r0w) / d.stride_w + 1 : 0;
    g.eh = (ph + r0h - P) / d.stride_h; g.ew = (pw + r0w - Q) / d.stride_w;   // exact divisions
    g.sh = g.sw = 1;
    const int T = g.Th * g.Tw;
    const long long pixels = (long long)d.n * g.mh * g.mw, m0 = (long long)blockIdx.x * BMT;
    if (m0 >= pixels) return;
    const int n0 = blockIdx.y * BNT;
    const int pitch = ord_row_pitch(T, QC), stage = (BMT + BNT) * pitch;
    const uint32_t smem0 = (uint32_t)__cvta_generic_to_shared(smem);
    Gather<BMT, THREADS> ga;
    Gather<BNT, THREADS> gb;
    if (T > 0) {
        gather_pixels(ga, g, QC >> 2, m0, pixels);
        gb.plan(T, QC >> 2, [&](int row, int tap) {
            const int a = tap / g.Tw, c = n0 + row;
            const int kt = (d.kh - 1 - r0h - d.stride_h * a) * d.kw + d.kw - 1 - r0w - d.stride_w * (tap - a * g.Tw);
            return c < d.c ? (kt * d.c + c) * d.o : -1;
        });
    }
    auto load_stage = [&](int q0, int buf) {
        const uint32_t as = smem0 + 4u * (uint32_t)(buf * stage);
        ga.load(as, pitch, T, dy, q0, QC, d.o, vec);
        gb.load(as + 4u * (uint32_t)(BMT * pitch), pitch, T, k, q0, QC, d.o, vec);
        cp_async_commit();
    };
    const int tx = tid % TX, ty = tid / TX;
    float tot[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) tot[i][j] = 0.f;
    if (T > 0) {
#pragma unroll
        for (int s = 0; s < STAGES - 1; ++s) {
            if (s * QC < d.o) load_stage(s * QC, s);
            else cp_async_commit();
        }
        int buf = 0, next = STAGES - 1;
        for (int q0 = 0; q0 < d.o; q0 += QC) {
            if (q0 + (STAGES - 1) * QC < d.o) load_stage(q0 + (STAGES - 1) * QC, next);
            else cp_async_commit();
            next = next + 1 == STAGES ? 0 : next + 1;
            cp_async_wait<STAGES - 1>();
            __syncthreads();
            const float *as[TM], *bs[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) as[i] = smem + buf * stage + (ty + i * TY) * pitch;
#pragma unroll
            for (int j = 0; j < TN; ++j) bs[j] = smem + buf * stage + (BMT + tx + j * TX) * pitch;
            const int quads = min(QC, d.o - q0 + 3) >> 2;
            auto chunk = [&](auto taps_c) {
                constexpr int TC = decltype(taps_c)::value;   // taps at compile time, 0: run time
                for (int q = 0; q < quads; ++q) {
                    float val[TM][TN][4];
#pragma unroll
                    for (int i = 0; i < TM; ++i)
#pragma unroll
                        for (int j = 0; j < TN; ++j) val[i][j][0] = val[i][j][1] = val[i][j][2] = val[i][j][3] = 0.f;
                    // U taps: operands first, then their products and sums
                    auto taps = [&](auto u_c) {
                        constexpr int U = decltype(u_c)::value;
                        float a[U][TM][4], b[U][TN][4];
#pragma unroll
                        for (int u = 0; u < U; ++u) {
#pragma unroll
                            for (int i = 0; i < TM; ++i) lds_vec<4>(as[i] + 4 * u, a[u][i]);
#pragma unroll
                            for (int j = 0; j < TN; ++j) lds_vec<4>(bs[j] + 4 * u, b[u][j]);
                        }
#pragma unroll
                        for (int i = 0; i < TM; ++i) as[i] += 4 * U;
#pragma unroll
                        for (int j = 0; j < TN; ++j) bs[j] += 4 * U;
#pragma unroll
                        for (int u = 0; u < U; ++u)
#pragma unroll
                            for (int i = 0; i < TM; ++i)
#pragma unroll
                                for (int j = 0; j < TN; ++j)
#pragma unroll
                                    for (int f = 0; f < 4; ++f)
                                        val[i][j][f] = __fadd_rn(val[i][j][f], __fmul_rn(a[u][i][f], b[u][j][f]));
                    };
                    if constexpr (TC > 0) {
#pragma unroll
                        for (int t = 0; t + 1 < TC; t += 2) taps(std::integral_constant<int, 2>());
                        if constexpr (TC % 2 != 0) taps(std::integral_constant<int, 1>());
                    } else {
                        for (int t = 0; t < T; ++t) taps(std::integral_constant<int, 1>());
                    }
                    // filters beyond the last are zero-filled: they add +0
#pragma unroll
                    for (int u = 0; u < 4; ++u)
#pragma unroll
                        for (int i = 0; i < TM; ++i)
#pragma unroll
                            for (int j = 0; j < TN; ++j) tot[i][j] = __fadd_rn(tot[i][j], val[i][j][u]);
                }
            };
            switch (T) {   // the classes of 5 x 5 / stride 2 (and 3 x 3): taps unrolled
            case 4: chunk(std::integral_constant<int, 4>()); break;
            case 6: chunk(std::integral_constant<int, 6>()); break;
            case 9: chunk(std::integral_constant<int, 9>()); break;
            default: chunk(std::integral_constant<int, 0>()); break;
            }
            __syncthreads();
            buf = buf + 1 == STAGES ? 0 : buf + 1;
        }
    }
    if constexpr (!dx_again_inside(TM)) {
        if (any_nan(tot)) g_nan_seen = 1;
    } else if (any_nan(tot)) {
#pragma unroll 1
        for (int i = 0; i < TM * TN; ++i) {
            const int p = (int)m0 + ty + i / TN * TY, ch = n0 + tx + i % TN * TX;
            if (p >= pixels || ch >= d.c) continue;
            const int line = p / g.mw, n = line / g.mh, r0 = line % g.mh, c0 = p % g.mw;
            float total = 0.f;
#pragma unroll 1
            for (int o = 0; o < d.o; ++o) {
                float v = 0.f;
#pragma unroll 1
                for (int t = 0; t < T; ++t) {
                    const int a = t / g.Tw, b = t % g.Tw, r = r0 + g.eh + a, c = c0 + g.ew + b;
                    const int kt = (d.kh - 1 - r0h - d.stride_h * a) * d.kw + d.kw - 1 - r0w - d.stride_w * b;
                    if (r >= 0 && r < d.ho && c >= 0 && c < d.wo)
                        v = __fadd_rn(v, __fmul_rn(__ldg(dy + ((n * d.ho + r) * d.wo + c) * d.o + o), __ldg(k + (kt * d.c + ch) * d.o + o)));
                }
                total = __fadd_rn(total, v);
            }
            const size_t idx = ((size_t)((n * d.h + r0 * d.stride_h + ph) * d.w) + c0 * d.stride_w + pw) * d.c + ch;
            dx[idx] = epilogue_apply(ep, total, idx, ch);
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const long long p = m0 + ty + i * TY;
        if (p >= pixels) continue;
        const int jj = (int)(p % g.mw);
        const long long t = p / g.mw;
        const size_t pix = ((size_t)(t / g.mh) * d.h + (size_t)(t % g.mh) * d.stride_h + ph) * d.w + (size_t)jj * d.stride_w + pw;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int ch = n0 + tx + j * TX;
            if (ch >= d.c) continue;
            const size_t idx = pix * d.c + ch;
            dx[idx] = epilogue_apply(ep, tot[i][j], idx, ch);
        }
    }
}

// ---- kernel gradient as an ordered GEMM -------------------------------------------------------------------
// dk[(tap, c), o] over K = (image outermost, output pixel innermost): the pixels of an image are summed
// first, the images' sums added in order.  Rows are (tap, channel) pairs, so a 3-channel layer fills its
// tiles as well as a 256-channel one.  Both operands are contiguous along the tile axes: a stage is KP pixels,
// A as [pixel][row] (16-byte copies where the channel count allows), B as [pixel][filter].  GROUPS thread groups
// of a block take every GROUPS-th image each and hand their sums over in shared memory, where the first group adds
// them in image order: more of the GPU for layers with few weights, same bits.
template <int TM, int TN, int TX, int TY, int STAGES, int GROUPS>
__global__ void __launch_bounds__(TX * TY * GROUPS)
conv_ordered_dk_kernel(const float* __restrict__ x, const float* __restrict__ dy, float* __restrict__ dk,
                       const dcg_conv_desc d, const int vec_a, const int vec_b)
{
    constexpr int BMT = TM * TY, BNT = TN * TX, THREADS = TX * TY, KP = 32, LDA = ord_pitch(BMT), LDB = ord_pitch(BNT);
    constexpr int STAGE = KP * (LDA + LDB);
    extern __shared__ __align__(16) float smem[];
    pdl_enter();
    const int group = threadIdx.x / THREADS, tid = threadIdx.x % THREADS;
    const int M = d.kh * d.kw * d.c, P = d.ho * d.wo;
    const int m0 = blockIdx.x * BMT, n0 = blockIdx.y * BNT;
    float* mine = smem + group * STAGES * STAGE;
    const uint32_t mine0 = (uint32_t)__cvta_generic_to_shared(mine);
    // gather roles: one row quad (or row) of A and one filter quad (or filter) of B, every few pixels
    const int aw = vec_a ? 4 : 1, bw = vec_b ? 4 : 1;
    const int acols = BMT / aw, bcols = BNT / bw;
    const int ac = (tid % acols) * aw, ar0 = tid / acols, arstep = THREADS / acols;
    const int bc = (tid % bcols) * bw, br0 = tid / bcols, brstep = THREADS / bcols;
    const int m = m0 + ac;
    const bool m_in = m < M, o_in = n0 + bc < d.o;
    const int c = m % d.c, tap = m / d.c, dh = (tap / d.kw) - d.pad_top, dw = (tap % d.kw) - d.pad_left;
    auto load_stage = [&](int n, int p0, int buf) {
        if (n < d.n) {
            const uint32_t as = mine0 + 4u * (uint32_t)(buf * STAGE), bs = as + 4u * (uint32_t)(KP * LDA);
            const int rows = min(KP, P - p0);
            int r = ar0, a = (p0 + ar0) / d.wo, b = (p0 + ar0) % d.wo;
            const float* xn = x + (long long)n * d.h * d.w * d.c + c;
            for (; r < rows; r += arstep) {
                const int h = d.stride_h * a + dh, w = d.stride_w * b + dw;
                const bool in = m_in && h >= 0 && h < d.h && w >= 0 && w < d.w;
                const float* s = in ? xn + ((long long)h * d.w + w) * d.c : x;
                const uint32_t dst = as + 4u * (uint32_t)(r * LDA + ac);
                if (vec_a) cp_async16(dst, s, in);
                else cp_async4(dst, s, in);
                b += arstep;
                while (b >= d.wo) { b -= d.wo; ++a; }
            }
            const float* g = dy + ((long long)n * P + p0) * d.o + n0 + bc;
            for (r = br0; r < rows; r += brstep) {
                const float* s = o_in ? g + (long long)r * d.o : dy;
                const uint32_t dst = bs + 4u * (uint32_t)(r * LDB + bc);
                if (vec_b) cp_async16(dst, s, o_in);
                else cp_async4(dst, s, o_in);
            }
        }
        cp_async_commit();
    };
    const int tx = tid % TX, ty = tid / TX;
    float val[TM][TN], tot[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) val[i][j] = tot[i][j] = 0.f;
    const int rounds = (d.n + GROUPS - 1) / GROUPS, chunks = (P + KP - 1) / KP;
    // stages run through the images of this group one after the other
    int ln = group, lck = 0;
    auto load_next = [&](int b) {
        load_stage(ln, lck * KP, b);
        if (++lck == chunks) { lck = 0; ln += GROUPS; }
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) load_next(s);
    int buf = 0, next = STAGES - 1;
    for (int rd = 0; rd < rounds; ++rd) {
        const int n = rd * GROUPS + group;
        for (int ck = 0; ck < chunks; ++ck) {
            load_next(next);
            next = next + 1 == STAGES ? 0 : next + 1;
            cp_async_wait<STAGES - 1>();
            __syncthreads();
            if (n < d.n) {
                const float* as = mine + buf * STAGE + ty * TM;
                const float* bs = mine + buf * STAGE + KP * LDA + tx * TN;
                const int rows = min(KP, P - ck * KP);
                constexpr int U = TM * TN <= 4 ? 8 : 4;
                int r = 0;
                for (; r + U <= rows; r += U) {
                    float a[U][TM], b[U][TN];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        lds_vec<TM>(as + u * LDA, a[u]);
                        lds_vec<TN>(bs + u * LDB, b[u]);
                    }
                    as += U * LDA;
                    bs += U * LDB;
#pragma unroll
                    for (int u = 0; u < U; ++u)
#pragma unroll
                        for (int i = 0; i < TM; ++i)
#pragma unroll
                            for (int j = 0; j < TN; ++j) val[i][j] = __fadd_rn(val[i][j], __fmul_rn(a[u][i], b[u][j]));
                }
                for (; r < rows; ++r) {
                    float a[TM], b[TN];
                    lds_vec<TM>(as, a);
                    lds_vec<TN>(bs, b);
                    as += LDA;
                    bs += LDB;
#pragma unroll
                    for (int i = 0; i < TM; ++i)
#pragma unroll
                        for (int j = 0; j < TN; ++j) val[i][j] = __fadd_rn(val[i][j], __fmul_rn(a[i], b[j]));
                }
            }
            __syncthreads();
            buf = buf + 1 == STAGES ? 0 : buf + 1;
        }
        if (GROUPS == 1) {
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) { tot[i][j] = __fadd_rn(tot[i][j], val[i][j]); val[i][j] = 0.f; }
        } else {
            float* red = smem + GROUPS * STAGES * STAGE;   // [group][item][thread]
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    red[(group * TM * TN + i * TN + j) * THREADS + tid] = val[i][j];
                    val[i][j] = 0.f;
                }
            __syncthreads();
            if (group == 0)
                for (int g = 0; g < GROUPS && rd * GROUPS + g < d.n; ++g)
#pragma unroll
                    for (int i = 0; i < TM; ++i)
#pragma unroll
                        for (int j = 0; j < TN; ++j)
                            tot[i][j] = __fadd_rn(tot[i][j], red[(g * TM * TN + i * TN + j) * THREADS + tid]);
            // the barrier of the next stage comes before anybody overwrites `red`
        }
    }
    if (group != 0) return;
    if constexpr (!dk_again_inside(TM, TN)) {
        if (any_nan(tot)) g_nan_seen = 1;
    } else if (any_nan(tot)) {
#pragma unroll 1
        for (int i = 0; i < TM * TN; ++i) {
            const int row = m0 + ty * TM + i / TN, o = n0 + tx * TN + i % TN;
            if (row >= M || o >= d.o) continue;
            const int t = row / d.c, q = row % d.c;
            float total = 0.f;
#pragma unroll 1
            for (int n = 0; n < d.n; ++n) {
                float v = 0.f;
#pragma unroll 1
                for (int p = 0; p < P; ++p) {
                    const int h = p / d.wo * d.stride_h + t / d.kw - d.pad_top, w = p % d.wo * d.stride_w + t % d.kw - d.pad_left;
                    if (h >= 0 && h < d.h && w >= 0 && w < d.w)
                        v = __fadd_rn(v, __fmul_rn(__ldg(x + ((n * d.h + h) * d.w + w) * d.c + q), __ldg(dy + (n * P + p) * d.o + o)));
                }
                total = __fadd_rn(total, v);
            }
            dk[(size_t)row * d.o + o] = total;
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int row = m0 + ty * TM + i;
        if (row >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int o = n0 + tx * TN + j;
            if (o < d.o) dk[(size_t)row * d.o + o] = tot[i][j];
        }
    }
}

// `cols` columns in tiles of `tile` where there are as many as to matter, `classes` parity classes: grid.y and grid.z.
bool ordered_ok(const dcg_conv_desc& d, int cols, int tile, long long classes = 1)
{
    if (cols > 65535 * tile || classes > 65535) return false;
    // element offsets are 32-bit
    const long long x = (long long)d.n * d.h * d.w * d.c, y = (long long)d.n * d.ho * d.wo * d.o, k = (long long)d.kh * d.kw * d.c * d.o;
    return d.kh * d.kw <= kOrdMaxTaps && x < (1ll << 31) && y < (1ll << 31) && k < (1ll << 31);
}
bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Behind an ordered launch of which some output has a tap outside the source.  An output that has replaced its gate stays as it is.
template <int KIND>
int nan_again(const float* a, const float* b, float* out, const dcg_conv_desc& d, const EpilogueArgs& ep, size_t total, cudaStream_t stream)
{
    const bool leaves = KIND == kOrdDx ? d.kh * d.kw * d.stride_h * d.stride_w > 1
                                       : d.pad_top > 0 || d.pad_left > 0 || (d.ho - 1) * d.stride_h + d.kh > d.h || (d.wo - 1) * d.stride_w + d.kw > d.w;
    if (!leaves || ep.gate == out) return DCG_OK;
    size_t blocks = (total + kThreads - 1) / kThreads;
    if (blocks > (size_t)sm_count()) blocks = sm_count();
    launch_pdl(conv_nan_again_kernel<KIND>, (unsigned)blocks, kThreads, 0, stream, a, b, out, d, ep, total);
    DCG_CUDA(cudaGetLastError());   // not counted: no operator's launch but a look behind one
    return DCG_OK;
}

// Channels per stage: kOrdQuads words of `taps` each, no more than there are.
int ord_channels(int taps, int contracted)
{
    int qc = kOrdQuads / (taps > 0 ? taps : 1) * 4;
    const int all = (contracted + 3) / 4 * 4;
    if (qc > 32) qc = 32;
    if (qc > all) qc = all;
    return qc < 4 ? 4 : qc;
}

template <int TM, int TN, int TX, int TY, int STAGES, int U>
int launch_ordered_fwd_taps(const dcg_conv_desc& d, const float* x, const float* k, float* y, const EpilogueArgs& ep, cudaStream_t stream)
{
    constexpr int BMT = TM * TY, BNT = TN * TX;
    static OncePerDevice once;
    DCG_CUDA(allow_smem(once, conv_ordered_fwd_kernel<TM, TN, TX, TY, STAGES, U>, kOrdSmem));
    const int taps = d.kh * d.kw, qc = ord_channels(taps, d.c);
    const size_t smem = (size_t)STAGES * (BMT * ord_row_pitch(taps, qc) + qc * taps * ord_pitch(BNT)) * sizeof(float);
    const long long pixels = (long long)d.n * d.ho * d.wo;
    const dim3 grid((unsigned)((pixels + BMT - 1) / BMT), (unsigned)((d.o + BNT - 1) / BNT));
    launch_pdl(conv_ordered_fwd_kernel<TM, TN, TX, TY, STAGES, U>, grid, TX * TY, smem, stream, x, k, y, d, ep, qc,
               d.c % 4 == 0 && aligned16(x) ? 1 : 0, d.o % 4 == 0 && aligned16(k) ? 1 : 0);
    DCG_LAUNCH_CHECK("conv_ordered_fwd_kernel");
    return nan_again<kOrdFwd>(x, k, y, d, ep, (size_t)pixels * d.o, stream);
}

template <int TM, int TN, int TX, int TY, int STAGES>
int launch_ordered_fwd_tile(const dcg_conv_desc& d, const float* x, const float* k, float* y, const EpilogueArgs& ep, cudaStream_t stream)
{
    const int taps = d.kh * d.kw;
    if (TM * TN <= 4 && taps == 25) return launch_ordered_fwd_taps<TM, TN, TX, TY, STAGES, TM * TN <= 4 ? 25 : 5>(d, x, k, y, ep, stream);
    if (taps % 5 == 0) return launch_ordered_fwd_taps<TM, TN, TX, TY, STAGES, 5>(d, x, k, y, ep, stream);
    if (taps % 4 == 0) return launch_ordered_fwd_taps<TM, TN, TX, TY, STAGES, 4>(d, x, k, y, ep, stream);
    if (taps % 3 == 0) return launch_ordered_fwd_taps<TM, TN, TX, TY, STAGES, 3>(d, x, k, y, ep, stream);
    return launch_ordered_fwd_taps<TM, TN, TX, TY, STAGES, 1>(d, x, k, y, ep, stream);
}

template <int TM, int TN, int TX, int TY, int STAGES>
int launch_ordered_dx_tile(const dcg_conv_desc& d, const float* dy, const float* k, float* dx, const EpilogueArgs& ep, cudaStream_t stream)
{
    constexpr int BMT = TM * TY, BNT = TN * TX;
    static OncePerDevice once;
    DCG_CUDA(allow_smem(once, conv_ordered_dx_kernel<TM, TN, TX, TY, STAGES>, kOrdSmem));
    const int mh = (d.h + d.stride_h - 1) / d.stride_h, mw = (d.w + d.stride_w - 1) / d.stride_w;   // of the largest class
    const int taps = ((d.kh + d.stride_h - 1) / d.stride_h) * ((d.kw + d.stride_w - 1) / d.stride_w);
    const int qc = ord_channels(taps, d.o);
    const size_t smem = (size_t)STAGES * (BMT + BNT) * ord_row_pitch(taps, qc) * sizeof(float);
    const dim3 grid((unsigned)(((long long)d.n * mh * mw + BMT - 1) / BMT), (unsigned)((d.c + BNT - 1) / BNT),
                    (unsigned)(d.stride_h * d.stride_w));
    launch_pdl(conv_ordered_dx_kernel<TM, TN, TX, TY, STAGES>, grid, TX * TY, smem, stream, dy, k, dx, d, ep, qc,
               d.o % 4 == 0 && aligned16(dy) && aligned16(k) ? 1 : 0);
    DCG_LAUNCH_CHECK("conv_ordered_dx_kernel");
    return dx_again_inside(TM) ? DCG_OK : nan_again<kOrdDx>(dy, k, dx, d, ep, (size_t)d.n * d.h * d.w * d.c, stream);
}

// Tile choice by outputs per lane of the GPU (SMs x 128): the wider the thread tile the fewer instructions an output
// costs per K step, but a scheduler needs a few warps to hide the chain of dependent adds and the shared-memory
// latency: with one it issues an instruction every three clocks.  Forward of 8 images: 64 -> 128 75 -> 68 us with 2 x 4
// outputs per thread (4 x 4: 92 and more), 256 -> 512 127 -> 121 with 2 x 2; 12 -> 32 of 4 images of 33 x 47 35 -> 18.
constexpr double kOrdWide = 32, kOrdNormal = 5, kOrdFew = 3, kOrdDkGrouped = 2;

double outputs_per_lane(double outputs) { return outputs / (128.0 * sm_count()); }

int launch_ordered_fwd(const dcg_conv_desc& d, const float* x, const float* k, float* y, const EpilogueArgs& ep, cudaStream_t stream)
{
    const double per_lane = outputs_per_lane((double)d.n * d.ho * d.wo * d.o);
    if (per_lane >= kOrdWide) return launch_ordered_fwd_tile<4, 4, 16, 16, 2>(d, x, k, y, ep, stream);
    if (per_lane >= 2 * kOrdNormal) return launch_ordered_fwd_tile<2, 4, 16, 16, 2>(d, x, k, y, ep, stream);
    if (per_lane >= kOrdNormal) return launch_ordered_fwd_tile<2, 2, 16, 16, 2>(d, x, k, y, ep, stream);
    if (per_lane >= kOrdFew) return launch_ordered_fwd_tile<2, 2, 16, 8, 4>(d, x, k, y, ep, stream);
    return launch_ordered_fwd_tile<1, 2, 8, 16, 4>(d, x, k, y, ep, stream);
}

int launch_ordered_dx(const dcg_conv_desc& d, const float* dy, const float* k, float* dx, const EpilogueArgs& ep, cudaStream_t stream)
{
    const double per_lane = outputs_per_lane((double)d.n * d.h * d.w * d.c);
    if (d.c <= 4) return launch_ordered_dx_tile<1, 4, 1, 128, 2>(d, dy, k, dx, ep, stream);   // RGB images: a pixel per thread
    if (per_lane >= kOrdWide) return launch_ordered_dx_tile<4, 2, 16, 16, 2>(d, dy, k, dx, ep, stream);
    if (per_lane >= kOrdNormal) return launch_ordered_dx_tile<2, 2, 16, 16, 2>(d, dy, k, dx, ep, stream);
    return launch_ordered_dx_tile<1, 2, 8, 16, 4>(d, dy, k, dx, ep, stream);
}

template <int TM, int TN, int TX, int TY, int STAGES, int GROUPS>
int launch_ordered_dk_tile(const dcg_conv_desc& d, const float* x, const float* dy, float* dk, cudaStream_t stream)
{
    constexpr int BMT = TM * TY, BNT = TN * TX;
    const size_t smem = (size_t)GROUPS * STAGES * 32 * (ord_pitch(BMT) + ord_pitch(BNT)) * 4 + (GROUPS > 1 ? (size_t)GROUPS * BMT * BNT * 4 : 0);
    static OncePerDevice once;
    DCG_CUDA(allow_smem(once, conv_ordered_dk_kernel<TM, TN, TX, TY, STAGES, GROUPS>, kOrdSmem));
    const int M = d.kh * d.kw * d.c;
    const dim3 grid((unsigned)((M + BMT - 1) / BMT), (unsigned)((d.o + BNT - 1) / BNT));
    launch_pdl(conv_ordered_dk_kernel<TM, TN, TX, TY, STAGES, GROUPS>, grid, TX * TY * GROUPS, smem, stream, x, dy, dk, d,
               d.c % 4 == 0 && aligned16(x) ? 1 : 0, d.o % 4 == 0 && aligned16(dy) ? 1 : 0);
    DCG_LAUNCH_CHECK("conv_ordered_dk_kernel");
    return dk_again_inside(TM, TN) ? DCG_OK : nan_again<kOrdDk>(x, dy, dk, d, EpilogueArgs{}, (size_t)M * d.o, stream);
}

int launch_ordered_dk(const dcg_conv_desc& d, const float* x, const float* dy, float* dk, cudaStream_t stream)
{
    // the images of a batch are parallel work as well (GROUPS); outputs per lane as above
    const double per_lane = (double)d.kh * d.kw * d.c * d.o / (128.0 * sm_count());
    if (per_lane >= kOrdWide) return launch_ordered_dk_tile<4, 4, 16, 16, 2, 1>(d, x, dy, dk, stream);
    if (per_lane < kOrdDkGrouped && d.n >= 8) return launch_ordered_dk_tile<1, 2, 4, 8, 4, 16>(d, x, dy, dk, stream);
    if (per_lane >= kOrdDkGrouped && d.n > 2) return launch_ordered_dk_tile<4, 4, 8, 8, 2, 4>(d, x, dy, dk, stream);
    return launch_ordered_dk_tile<2, 2, 8, 8, 4, 1>(d, x, dy, dk, stream);
}


// ---- one thread per output: kernels with many taps ----------------------------------------------------
__global__ void __launch_bounds__(kThreads)
conv_fwd_generic_kernel(const float* __restrict__ x, const float* __restrict__ k, float* __restrict__ y,
                        const dcg_conv_desc d, const EpilogueArgs ep, size_t total)
{
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const int o = (int)(idx % d.o);
    y[idx] = epilogue_apply(ep, fwd_sum(x, k, d, idx / d.o, o), idx, o);
}

__global__ void __launch_bounds__(kThreads)
conv_dx_generic_kernel(const float* __restrict__ dy, const float* __restrict__ k, float* __restrict__ dx,
                       const dcg_conv_desc d, const EpilogueArgs ep, size_t total)
{
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const int c = (int)(idx % d.c);
    dx[idx] = epilogue_apply(ep, dx_sum(dy, k, d, idx / d.c, c), idx, c);
}

__global__ void __launch_bounds__(kThreads)
conv_dk_generic_kernel(const float* __restrict__ x, const float* __restrict__ dy, float* __restrict__ dk,
                       const dcg_conv_desc d, size_t total)
{
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < total) dk[idx] = dk_sum(x, dy, d, idx / d.o, (int)(idx % d.o));
}

}  // namespace

int conv_fwd_generic(const dcg_conv_desc& d, const float* x, const float* k, float* y,
                     const EpilogueArgs& ep, cudaStream_t stream)
{
    const size_t total = (size_t)d.n * d.ho * d.wo * d.o;
    if (total == 0) return DCG_OK;
    if (ordered_ok(d, d.o, 64)) return launch_ordered_fwd(d, x, k, y, ep, stream);
    conv_fwd_generic_kernel<<<(unsigned)((total + kThreads - 1) / kThreads), kThreads, 0, stream>>>(
        x, k, y, d, ep, total);
    DCG_LAUNCH_CHECK("conv_fwd_generic_kernel");
    return DCG_OK;
}

int conv_dx_generic(const dcg_conv_desc& d, const float* dy, const float* k, float* dx,
                    const EpilogueArgs& ep, cudaStream_t stream)
{
    const size_t total = (size_t)d.n * d.h * d.w * d.c;
    if (total == 0) return DCG_OK;
    if (ordered_ok(d, d.c, 32, (long long)d.stride_h * d.stride_w)) return launch_ordered_dx(d, dy, k, dx, ep, stream);
    conv_dx_generic_kernel<<<(unsigned)((total + kThreads - 1) / kThreads), kThreads, 0, stream>>>(
        dy, k, dx, d, ep, total);
    DCG_LAUNCH_CHECK("conv_dx_generic_kernel");
    return DCG_OK;
}

int conv_dk_generic(const dcg_conv_desc& d, const float* x, const float* dy, float* dk,
                    cudaStream_t stream)
{
    const size_t total = (size_t)d.kh * d.kw * d.c * d.o;
    if (total == 0) return DCG_OK;
    if (ordered_ok(d, d.o, 64)) return launch_ordered_dk(d, x, dy, dk, stream);
    conv_dk_generic_kernel<<<(unsigned)((total + kThreads - 1) / kThreads), kThreads, 0, stream>>>(
        x, dy, dk, d, total);
    DCG_LAUNCH_CHECK("conv_dk_generic_kernel");
    return DCG_OK;
}

}  // namespace dcg

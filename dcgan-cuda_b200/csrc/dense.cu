// Dense-layer matrix products (src/gpu/matmul.cu:11-86): the generator's
// 100 -> 8192 projection, the discriminator's 8192 -> 1 head, and the MNIST MLP.
//
// These are small and HBM / latency bound (the largest operand is 3.3 MB), so they stay on CUDA cores.
// gemm_ordered_kernel accumulates each output over k in ascending order with unfused multiply / add - bit-identical to
// the reference CPU loops (src/cpu/ops.hxx:56-105,375-390); two shape specialists go with it: few outputs / long
// reduction (8192 -> 1), and tall output from a transposed operand (the head's weight gradient).
#include <cstdint>
#include <type_traits>

#include "colsum.cuh"
#include "common.cuh"

namespace dcg {
namespace {

constexpr int TPB = 256;

__device__ __forceinline__ void cp_async(uint32_t dst, const float* src, bool in, int bytes)
{
    const int n = in ? bytes : 0;   // 0: zero-fill
    if (bytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

// W consecutive floats of an operand tile
template <int W>
__device__ __forceinline__ void tile_read(const float* s, float (&v)[W])
{
    if constexpr (W == 4) {
        const float4 t = *reinterpret_cast<const float4*>(s);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else if constexpr (W == 2) {
        const float2 t = *reinterpret_cast<const float2*>(s);
        v[0] = t.x; v[1] = t.y;
    } else {
        v[0] = *s;
    }
}

// What follows the sum of an output: + bias[col], the value itself to `out`, an activation of it or its product with the
// activation gradient at gate[] to `out2` (same expressions as bias_act_kernel and act_grad_kernel).
struct DenseEpilogue {
    const float* bias;
    const float* gate;
    float* out2;
    int act;         // of out2: activation, or with `gate` the activation whose gradient gates
    float alpha;
    float* sums;     // TA only: column sums of B, as dcg_colsum adds them, by the first `sum_rows` rows of blocks
    ColsumTile sum;
    int sum_rows;
    bool out_dead;   // `out` need not be written (gemm_outer_kernel leaves it out)
};

// out[m,p] = A[m,n] B[n,p]: TM x TN outputs per thread, TX x TY threads per block, STAGES stages of KC reduction steps
// filled with cp.async.  TA / TB: the logical matrix is the transpose of the stored row-major one.  An operand whose
// reduction axis is contiguous keeps it so in shared memory ([row][k], four steps per 16-byte read), the other is
// [k][row].  What is beyond an edge is zero-filled; the zeros add +0 to the sums.
// Latency-bound at the sizes of this library: many small tiles and all loads of several stages in flight matter more than
// operand reuse (100 x 784 x 100: 160 us with one 64 x 64 tile per block and blocking loads).
template <bool TA, bool TB, int TM, int TN, int TX, int TY, int STAGES, int KC>
__global__ void __launch_bounds__(TX * TY)
gemm_ordered_kernel(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ out, const int m, const int n,
                    const int p, const DenseEpilogue e, const int vec_a, const int vec_b, const int vec_out)
{
    constexpr int BM = TM * TY, BN = TN * TX, THREADS = TX * TY;
    constexpr int LDA = TA ? BM + 4 : KC + 4, LDB = TB ? KC + 4 : BN + 4;
    constexpr int A_FLOATS = (TA ? KC : BM) * LDA, STAGE = A_FLOATS + (TB ? BN : KC) * LDB;
    extern __shared__ __align__(16) float smem[];
    pdl_enter();
    const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
    int block_row = blockIdx.y;
    if constexpr (TA && !TB) {
        if (block_row < e.sum_rows) {
            for (unsigned tile = block_row * gridDim.x + blockIdx.x; tile < e.sum.tiles; tile += e.sum_rows * gridDim.x) {
                if (e.sum.vec) colsum_tile_block<true>(b, e.sums, n, p, e.sum.order, e.sum.tile_shift, tile, THREADS, smem);
                else colsum_tile_block<false>(b, e.sums, n, p, e.sum.order, e.sum.tile_shift, tile, THREADS, smem);
                __syncthreads();
            }
            return;
        }
        block_row -= e.sum_rows;
    }
    const int row0 = block_row * BM, col0 = blockIdx.x * BN;
    const uint32_t smem0 = (uint32_t)__cvta_generic_to_shared(smem);

    // copies a tile of `inner` contiguous elements x `outer` lines, element (o, i) of the stored matrix at base[o * ld + i];
    // `inner` and the width of a copy are constants, so that a thread's places take shifts, not divisions
    auto copy_words = [&](auto inner_c, auto w_c, uint32_t dst, int pitch, const float* base, int o0, int i0, int outer, int limit, int o_end, int i_end) {
        constexpr int w = decltype(w_c)::value, per_line = decltype(inner_c)::value / w;
        for (int idx = tid; idx < outer * per_line; idx += THREADS) {
            const int o = idx / per_line, i = (idx - o * per_line) * w;
            if (i >= limit) continue;
            const bool in = o0 + o < o_end && i0 + i < i_end;
            cp_async(dst + 4u * (uint32_t)(o * pitch + i), in ? base + (size_t)(o0 + o) * i_end + i0 + i : base, in, 4 * w);
        }
    };
    auto copy_tile = [&](auto inner_c, uint32_t dst, int pitch, const float* base, int o0, int i0, int outer, int limit, int o_end, int i_end, int vec) {
        if (vec) copy_words(inner_c, std::integral_constant<int, 4>(), dst, pitch, base, o0, i0, outer, limit, o_end, i_end);
        else copy_words(inner_c, std::integral_constant<int, 1>(), dst, pitch, base, o0, i0, outer, limit, o_end, i_end);
    };
    using std::integral_constant;
    auto load_stage = [&](int k0, int buf) {
        if (k0 < n) {
            const uint32_t as = smem0 + 4u * (uint32_t)(buf * STAGE), bs = as + 4u * (uint32_t)A_FLOATS;
            const int kc = min(KC, (n - k0 + 3) & ~3);
            if (TA) copy_tile(integral_constant<int, BM>(), as, LDA, a, k0, row0, kc, BM, n, m, vec_a);
            else copy_tile(integral_constant<int, KC>(), as, LDA, a, row0, k0, BM, kc, m, n, vec_a);
            if (TB) copy_tile(integral_constant<int, KC>(), bs, LDB, b, col0, k0, BN, kc, p, n, vec_b);
            else copy_tile(integral_constant<int, BN>(), bs, LDB, b, k0, col0, kc, BN, n, p, vec_b);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) load_stage(s * KC, s);
    int buf = 0;
    for (int k0 = 0; k0 < n; k0 += KC) {
        load_stage(k0 + (STAGES - 1) * KC, (buf + STAGES - 1) % STAGES);
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 1) : "memory");
        __syncthreads();
        const float* as = smem + buf * STAGE + (TA ? ty * TM : ty * TM * LDA);
        const float* bs = smem + buf * STAGE + A_FLOATS + (TB ? tx * LDB : tx * TN);   // TB: columns tx, tx + TX, ...
        const int kc = min(KC, (n - k0 + 3) & ~3);
        // (one output to a thread: 32 steps of A^T B at a time, whose reads are single words; 100 x 2000 x 100 29 -> 26 us)
#pragma unroll (TA && !TB && TM * TN == 1 ? KC / 8 : KC / 16)
        for (int k = 0; k < kc; k += 4) {
            float av[4][TM], bv[4][TN];
            if (TA) {
#pragma unroll
                for (int u = 0; u < 4; ++u) tile_read<TM>(as + (k + u) * LDA, av[u]);
            } else {
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    float v[4];
                    tile_read<4>(as + i * LDA + k, v);
                    av[0][i] = v[0]; av[1][i] = v[1]; av[2][i] = v[2]; av[3][i] = v[3];
                }
            }
            if (TB) {
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    float v[4];
                    tile_read<4>(bs + j * TX * LDB + k, v);
                    bv[0][j] = v[0]; bv[1][j] = v[1]; bv[2][j] = v[2]; bv[3][j] = v[3];
                }
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u) tile_read<TN>(bs + (k + u) * LDB, bv[u]);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) acc[i][j] = __fadd_rn(acc[i][j], __fmul_rn(av[u][i], bv[u][j]));
        }
        __syncthreads();
        buf = (buf + 1) % STAGES;
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int r = row0 + ty * TM + i;
        if (r >= m) continue;
        if constexpr (!TB && TN == 4) {
            const int c = col0 + tx * TN;
            if (vec_out && !e.out2) {   // whole rows of 16-byte words
                if (c >= p) continue;
                float4 v = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
                if (e.bias) {
                    const float4 w = __ldg(reinterpret_cast<const float4*>(e.bias + c));
                    v.x = __fadd_rn(v.x, w.x); v.y = __fadd_rn(v.y, w.y); v.z = __fadd_rn(v.z, w.z); v.w = __fadd_rn(v.w, w.w);
                }
                *reinterpret_cast<float4*>(out + (size_t)r * p + c) = v;
                continue;
            }
        }
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int c = col0 + (TB ? tx + j * TX : tx * TN + j);
            if (c >= p) continue;
            const size_t idx = (size_t)r * p + c;
            float v = acc[i][j];
            if (e.bias) v = __fadd_rn(v, __ldg(e.bias + c));
            out[idx] = v;
            if (e.out2) e.out2[idx] = e.gate ? act_grad_apply(__ldg(e.gate + idx), v, e.act, e.alpha) : act_apply(v, e.act, e.alpha);
        }
    }
}

// Outer product of a column and a row (n == 1, whichever way the operands are stored: the input gradient of the head, 64 x 1
// times 1 x 8192, weight gradients of one row): four columns per thread, nothing to stage.  Memory-bound: the gate is read and both outputs written once.
__global__ void __launch_bounds__(TPB)
gemm_outer_kernel(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ out, const size_t m, const size_t p4,
                  const DenseEpilogue e)
{
    pdl_enter();
    const size_t total = m * p4, stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        const size_t r = i / p4, c4 = i - r * p4;
        const float av = __ldg(a + r);
        const float4 bv = __ldg(reinterpret_cast<const float4*>(b) + c4);
        float v[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = __fadd_rn(0.f, __fmul_rn(av, v[u]));
        if (e.bias) {
            const float4 w = __ldg(reinterpret_cast<const float4*>(e.bias) + c4);
            v[0] = __fadd_rn(v[0], w.x); v[1] = __fadd_rn(v[1], w.y); v[2] = __fadd_rn(v[2], w.z); v[3] = __fadd_rn(v[3], w.w);
        }
        if (!e.out_dead) reinterpret_cast<float4*>(out)[i] = make_float4(v[0], v[1], v[2], v[3]);
        if (e.out2) {
            if (e.gate) {
                const float4 g = __ldg(reinterpret_cast<const float4*>(e.gate) + i);
                v[0] = act_grad_apply(g.x, v[0], e.act, e.alpha); v[1] = act_grad_apply(g.y, v[1], e.act, e.alpha);
                v[2] = act_grad_apply(g.z, v[2], e.act, e.alpha); v[3] = act_grad_apply(g.w, v[3], e.act, e.alpha);
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = act_apply(v[u], e.act, e.alpha);
            }
            reinterpret_cast<float4*>(e.out2)[i] = make_float4(v[0], v[1], v[2], v[3]);
        }
    }
}

// One thread per output, 64-bit indexes: axes of 2^30 and more, which the tiles' 32-bit ones do not hold.  Same sums.
template <bool TA, bool TB>
__global__ void __launch_bounds__(TPB)
gemm_long_axis_kernel(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ out, const size_t m, const size_t n,
                      const size_t p, const DenseEpilogue e)
{
    pdl_enter();
    const size_t total = m * p, stride = (size_t)gridDim.x * blockDim.x;
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += stride) {
        const size_t r = idx / p, c = idx - r * p;
        float v = 0.f;
#pragma unroll 8
        for (size_t k = 0; k < n; ++k)
            v = __fadd_rn(v, __fmul_rn(__ldg(TA ? a + k * m + r : a + r * n + k), __ldg(TB ? b + c * n + k : b + k * p + c)));
        if (e.bias) v = __fadd_rn(v, __ldg(e.bias + c));
        out[idx] = v;
        if (e.out2) e.out2[idx] = e.gate ? act_grad_apply(__ldg(e.gate + idx), v, e.act, e.alpha) : act_apply(v, e.act, e.alpha);
    }
}

// One block per output element, for m*p small and n long: out = A[m,n] B[n,p] (+bias).
// Thread t adds elements t, t+256, ... in ascending order; the 256 thread sums are then added
// in a fixed tree, so the result is independent of scheduling.
__global__ void __launch_bounds__(TPB)
gemm_long_k_kernel(const float* __restrict__ a, const float* __restrict__ b,
                   const float* __restrict__ bias, float* __restrict__ out,
                   size_t m, size_t n, size_t p)
{
    pdl_enter();
    __shared__ float part[TPB];
    const size_t o = blockIdx.x;
    const size_t r = o / p, c = o % p;
    const float* ar = a + r * n;
    float s = 0.f;
    size_t k = threadIdx.x;
    for (; k + 3 * TPB < n; k += 4 * TPB) {
        const float a0 = __ldg(ar + k), a1 = __ldg(ar + k + TPB), a2 = __ldg(ar + k + 2 * TPB), a3 = __ldg(ar + k + 3 * TPB);
        const float b0 = __ldg(b + k * p + c), b1 = __ldg(b + (k + TPB) * p + c);
        const float b2 = __ldg(b + (k + 2 * TPB) * p + c), b3 = __ldg(b + (k + 3 * TPB) * p + c);
        s = fmaf(a0, b0, s); s = fmaf(a1, b1, s); s = fmaf(a2, b2, s); s = fmaf(a3, b3, s);
    }
    for (; k < n; k += TPB) s = fmaf(__ldg(ar + k), __ldg(b + k * p + c), s);
    part[threadIdx.x] = s;
    __syncthreads();
    for (int h = TPB / 2; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) part[threadIdx.x] += part[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[o] = bias ? part[0] + __ldg(bias + c) : part[0];
}

// Tall output with a handful of columns from a transposed left operand (the discriminator head's
// weight gradient, x^T dy): out[r,c] = sum_k A^T[k,r] B[k,c]; one thread per output, loads
// coalesced along r, k ascending, unfused.
__global__ void __launch_bounds__(TPB)
gemm_tall_tn_kernel(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ out,
                    size_t m, size_t n, size_t p)
{
    pdl_enter();
    const size_t o = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= m * p) return;
    const size_t c = o / m, r = o % m;   // r fastest across threads: coalesced reads of A^T
    float s = 0.f;
    size_t k = 0;
    for (; k + 32 <= n; k += 32) {
        float av[32], bw[32];
#pragma unroll
        for (int u = 0; u < 32; ++u) { av[u] = __ldg(a + (k + u) * m + r); bw[u] = __ldg(b + (k + u) * p + c); }
#pragma unroll
        for (int u = 0; u < 32; ++u) s = __fadd_rn(s, __fmul_rn(av[u], bw[u]));
    }
    for (; k < n; ++k) s = __fadd_rn(s, __fmul_rn(__ldg(a + k * m + r), __ldg(b + k * p + c)));
    out[r * p + c] = s;
}

bool aligned16(const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; }

// Column sums that fit a block of any tile.
constexpr unsigned kSumSlabs = 32;
constexpr size_t kSumSmem = 8192;   // 512 lanes of 16 bytes

template <bool TA, bool TB, int TM, int TN, int TX, int TY, int STAGES, int KC = 64>
int launch_tile(const float* a, const float* b, float* out, size_t m, size_t n, size_t p, DenseEpilogue e, cudaStream_t stream)
{
    constexpr int BM = TM * TY, BN = TN * TX;
    constexpr size_t smem = (size_t)STAGES * ((TA ? KC * (BM + 4) : BM * (KC + 4)) + (TB ? BN * (KC + 4) : KC * (BN + 4))) * sizeof(float);
    static OncePerDevice once;
    DCG_CUDA(allow_smem(once, gemm_ordered_kernel<TA, TB, TM, TN, TX, TY, STAGES, KC>, smem));
    dim3 grid((unsigned)((p + BN - 1) / BN), (unsigned)((m + BM - 1) / BM));
    static_assert(smem >= kSumSmem && TX * TY <= 256, "the column sums run in the same blocks");
    if (e.sums) {   // a block each for the column tiles, up to 32: they are not to crowd the others on some of the SMs
        colsum_fit(e.sum, TX * TY);
        const int rows = (int)((e.sum.tiles + grid.x - 1) / grid.x), most = grid.x >= 32 ? 1 : (int)(32 / grid.x);
        e.sum_rows = rows < most ? rows : most;
        grid.y += e.sum_rows;
    }
    const int vec_a = (TA ? m : n) % 4 == 0 && aligned16(a), vec_b = (TB ? n : p) % 4 == 0 && aligned16(b);
    const int vec_out = p % 4 == 0 && aligned16(out) && aligned16(e.bias);
    const auto kernel = gemm_ordered_kernel<TA, TB, TM, TN, TX, TY, STAGES, KC>;
    if (TM * TN < 16 || KC < 64) {
        launch_pdl(kernel, grid, TX * TY, smem, stream, a, b, out, (int)m, (int)n, (int)p, e, vec_a, vec_b, vec_out);
    } else {
        // Long blocks, often fewer than SMs: launched while the previous kernel runs, they pile up on the SMs that it leaves free
        // and stay there (100 x 256 x 8192 38 us so, 27.7 after it; the gradients of a 784-512-10 classifier's step at 1000 rows
        // 271 and 164).  A launch that waits costs 0.3 us.
        kernel<<<grid, TX * TY, smem, stream>>>(a, b, out, (int)m, (int)n, (int)p, e, vec_a, vec_b, vec_out);
    }
    DCG_LAUNCH_CHECK("gemm_ordered_kernel");
    return DCG_OK;
}

// Tile choice by outputs per lane of the GPU, as for the ordered convolutions: few outputs go one to a thread over as many
// blocks as there are, with four stages in flight.  A handful of rows (a small batch through the generator's
// projection) gets flat tiles, so that few of its threads idle.
template <bool TA, bool TB>
int launch_ordered(const float* a, const float* b, float* out, size_t m, size_t n, size_t p, const DenseEpilogue& e, cudaStream_t stream)
{
    DCG_CHECK_ARG((m + 3) / 4 <= 65535u * 16, "dense: %zu rows are too many", m);
    if (!e.sums && n == 1 && p % 4 == 0 && aligned16(b) && aligned16(out) && aligned16(e.bias) && aligned16(e.gate) && aligned16(e.out2)) {
        size_t blocks = (m * (p / 4) + TPB - 1) / TPB;
        const size_t cap = (size_t)sm_count() * 8;
        if (blocks > cap) blocks = cap;
        launch_pdl(gemm_outer_kernel, (unsigned)blocks, TPB, 0, stream, a, b, out, m, p / 4, e);
        DCG_LAUNCH_CHECK("gemm_outer_kernel");
        return DCG_OK;
    }
    if (n >= (1u << 30) || p >= (1u << 30)) {
        size_t blocks = (m * p + TPB - 1) / TPB;
        const size_t cap = (size_t)sm_count() * 16;
        if (blocks > cap) blocks = cap;
        launch_pdl(gemm_long_axis_kernel<TA, TB>, (unsigned)blocks, TPB, 0, stream, a, b, out, m, n, p, e);
        DCG_LAUNCH_CHECK("gemm_long_axis_kernel");
        return DCG_OK;
    }
    const double per_lane = (double)m * (double)p / (128.0 * sm_count());
    if (m <= 8 && p >= 512) return launch_tile<TA, TB, 1, 1, 32, 8, 3>(a, b, out, m, n, p, e, stream);
    // a few reduction steps: shorter lines to walk through, the rest is stores (784 x 2 x 512 2.8 us, 4.8 with 64 steps a stage;
    // 4096 x 10 x 4096 29 and 58)
    if (per_lane >= 20 && n <= 16) return launch_tile<TA, TB, 4, 4, 16, 16, 2, 16>(a, b, out, m, n, p, e, stream);
    if (per_lane >= 20) return launch_tile<TA, TB, 4, 4, 16, 16, 2>(a, b, out, m, n, p, e, stream);
    if (per_lane >= 5) return launch_tile<TA, TB, 2, 2, 16, 16, 3>(a, b, out, m, n, p, e, stream);
    // Where 16 x 16 tiles would leave half of the SMs without a block, smaller ones; each sum is one chain of K steps, so what
    // counts is how few warps share an SM and, for long ones, how many steps there are between two barriers (100 x 784 x 100:
    // 11.8 us as 16 x 16 tiles, 9.7 as 8 x 16 of 128 steps; 100 x 100 x 10 2.9 as 8 x 8)
    if (per_lane < 1 && n >= 512) return launch_tile<TA, TB, 1, 1, 8, 16, 4, 128>(a, b, out, m, n, p, e, stream);
    if (per_lane < 1) return launch_tile<TA, TB, 1, 1, 8, 8, 4>(a, b, out, m, n, p, e, stream);
    // (rows of A^T are contiguous: two to a thread are one read; 784 x 100 x 100 5.3 -> 4.4 us)
    if (TA && per_lane >= 2) return launch_tile<TA, TB, 2, 1, 16, 8, 3>(a, b, out, m, n, p, e, stream);
    return launch_tile<TA, TB, 1, 1, 16, 16, 4>(a, b, out, m, n, p, e, stream);
}

int matmul_nn(const float* a, const float* b, float* out, size_t m, size_t n, size_t p, const DenseEpilogue& e, cudaStream_t stream)
{
    if (m * p <= 4096 && n >= 1024 && !e.out2) {
        launch_pdl(gemm_long_k_kernel, (unsigned)(m * p), TPB, 0, stream, a, b, e.bias, out, m, n, p);
        DCG_LAUNCH_CHECK("gemm_long_k_kernel");
        return DCG_OK;
    }
    return launch_ordered<false, false>(a, b, out, m, n, p, e, stream);
}

}  // namespace

// dcg_matmul followed by an activation of its result as one launch (node fusion of the backend).  Not for the shapes of
// gemm_long_k_kernel: returns 1 there.
int matmul_act(const float* a, const float* b, const float* bias, float* out, size_t m, size_t n, size_t p, int act, float alpha,
               float* act_out, cudaStream_t stream)
{
    if (m * p <= 4096 && n >= 1024) return 1;
    DCG_CHECK_ARG(a && b && out && act_out && m > 0 && n > 0 && p > 0, "matmul_act: bad arguments");
    return matmul_nn(a, b, out, m, n, p, DenseEpilogue{bias, nullptr, act_out, act, alpha}, stream);
}

// dcg_matmul_nt followed by dcg_act_grad(gate, out) -> gated_out as one launch (node fusion of the backend).  `out_dead`: nobody
// reads `out`.
int matmul_nt_gated(const float* a, const float* b, float* out, size_t m, size_t n, size_t p, const float* gate,
                    float* gated_out, int gate_act, float gate_alpha, bool out_dead, cudaStream_t stream)
{
    DCG_CHECK_ARG(a && b && out && gate && gated_out && m > 0 && n > 0 && p > 0, "matmul_nt_gated: bad arguments");
    DenseEpilogue e{nullptr, gate, gated_out, gate_act, gate_alpha};
    e.out_dead = out_dead;
    return launch_ordered<false, true>(a, b, out, m, n, p, e, stream);
}

// dcg_matmul_tn and the column sums of its right operand as one launch (node fusion of the backend): the weight and the bias
// gradient of a dense layer, both bit for bit.  Blocks of their own add the columns beside those of the product, which take as
// long or longer: 100 x 784 x 100 4.1 us with and without them, 2.3 for the sums by themselves.  Not for the shapes of
// gemm_tall_tn_kernel, nor for more rows than a block adds up (1024 where a column tile is 32 wide): returns 1 there.
int matmul_tn_sums(const float* a, const float* b, float* out, size_t m, size_t n, size_t p, float* sums, cudaStream_t stream)
{
    if ((p <= 8 && m >= 1024) || m > (1u << 20) || p >= (1u << 30)) return 1;
    DCG_CHECK_ARG(a && b && out && sums && m > 0 && n > 0 && p > 0, "matmul_tn_sums: bad arguments");
    DenseEpilogue e{};
    if (!colsum_order(n, p, aligned16(b), kSumSlabs, e.sum) || (e.sum.order.slabs << e.sum.order.lane_shift) * 16 > kSumSmem) return 1;
    e.sums = sums;
    return launch_ordered<true, false>(a, b, out, m, n, p, e, stream);
}

}  // namespace dcg

using namespace dcg;

extern "C" int dcg_matmul(const float* a, const float* b, const float* bias, float* out, size_t m,
                          size_t n, size_t p, dcg_stream_t stream)
{
    DCG_CHECK_ARG(a && b && out && m > 0 && n > 0 && p > 0, "dcg_matmul: bad arguments");
    return matmul_nn(a, b, out, m, n, p, DenseEpilogue{bias, nullptr, nullptr, DCG_ACT_NONE, 0.f}, as_stream(stream));
}

extern "C" int dcg_matmul_tn(const float* a, const float* b, float* out, size_t m, size_t n,
                             size_t p, dcg_stream_t stream)
{
    DCG_CHECK_ARG(a && b && out && m > 0 && n > 0 && p > 0, "dcg_matmul_tn: bad arguments");
    if (p <= 8 && m >= 1024) {
        launch_pdl(gemm_tall_tn_kernel, (unsigned)((m * p + 63) / 64), 64, 0, as_stream(stream), a, b, out, m, n, p);
        DCG_LAUNCH_CHECK("gemm_tall_tn_kernel");
        return DCG_OK;
    }
    return launch_ordered<true, false>(a, b, out, m, n, p, DenseEpilogue{}, as_stream(stream));
}

extern "C" int dcg_matmul_nt(const float* a, const float* b, float* out, size_t m, size_t n,
                             size_t p, dcg_stream_t stream)
{
    DCG_CHECK_ARG(a && b && out && m > 0 && n > 0 && p > 0, "dcg_matmul_nt: bad arguments");
    return launch_ordered<false, true>(a, b, out, m, n, p, DenseEpilogue{}, as_stream(stream));
}

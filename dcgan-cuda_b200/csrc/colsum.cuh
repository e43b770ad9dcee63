// Column sums of a few hundred rows inside one block: shared by the column-sum launch and by the dense weight gradient, whose
// launch sums the same output gradient.
#pragma once

#include "common.cuh"

namespace dcg {

// The order in which the rows of a column are added: slabs of rows_per_slab rows; within a slab `lanes` lanes (a power of two)
// take every lanes-th row each, at most four, and a halving tree adds the lanes; then slab s goes to lane s % lanes, and those
// are added in ascending order.  It follows from rows, columns and alignment alone, whoever computes it.
struct ColsumOrder {
    unsigned rows_per_slab, slabs;
    int lanes;
};

// How a block of `threads` threads computes it: `tile` column groups (float4s or floats; a power of two) at a time.
struct ColsumTile {
    ColsumOrder order;
    bool vec;
    int tile;
    unsigned tiles;   // column tiles
    size_t smem;      // bytes
};
// False where the order has more than `max_slabs` slabs or more than four rows per lane.
bool colsum_tile(size_t rows, size_t cols, bool aligned, int threads, unsigned max_slabs, ColsumTile& t);

#ifdef __CUDACC__
// Threads are [slab and lane][column group]: where a slab has few rows they run side by side, each with its rows in flight at
// once, instead of one slab after the other.  All threads of the block take part.
template <bool VEC>
__device__ __forceinline__ void colsum_tile_block(const float* __restrict__ a, float* __restrict__ out, const unsigned rows, const unsigned cols,
                                                  const ColsumOrder o, const int tile, const unsigned block, const int threads, float* smem)
{
    constexpr int W = VEC ? 4 : 1;
    const int width = tile * W, tid = threadIdx.x;
    const int tx = tid % tile, step = threads / tile, places = (int)o.slabs * o.lanes;
    const unsigned group = block * tile + tx, groups = cols / W;
    for (int v = tid / tile; v < places; v += step) {   // smem: [slab][lane][column]
        const unsigned s = v / o.lanes, r0 = s * o.rows_per_slab + v % o.lanes, r1 = min((s + 1) * o.rows_per_slab, rows);
        float acc[W];
#pragma unroll
        for (int q = 0; q < W; ++q) acc[q] = 0.f;
        if (group < groups) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const unsigned r = r0 + i * o.lanes;
                if (r < r1) {
                    if constexpr (VEC) {
                        const float4 x = __ldg(reinterpret_cast<const float4*>(a + (size_t)r * cols) + group);
                        acc[0] += x.x; acc[1] += x.y; acc[2] += x.z; acc[3] += x.w;
                    } else {
                        acc[0] += __ldg(a + (size_t)r * cols + group);
                    }
                }
            }
        }
#pragma unroll
        for (int q = 0; q < W; ++q) smem[v * width + tx * W + q] = acc[q];
    }
    __syncthreads();
    for (int h = o.lanes >> 1; h > 0; h >>= 1) {
        for (int i = tid; i < (int)o.slabs * h * width; i += threads) {
            const int u = i / width, at = (u / h * o.lanes + u % h) * width + i % width;
            smem[at] += smem[at + h * width];
        }
        __syncthreads();
    }
    for (int i = tid; i < width; i += threads) {
        const unsigned c = block * width + i;
        if (c >= cols) break;
        auto lane_sum = [&](int lane) {
            float r = smem[lane * o.lanes * width + i];
            for (unsigned s = lane + o.lanes; s < o.slabs; s += o.lanes) r += smem[s * o.lanes * width + i];
            return r;
        };
        float r = lane_sum(0);
        for (int lane = 1; lane < min(o.lanes, (int)o.slabs); ++lane) r += lane_sum(lane);
        out[c] = r;
    }
}
#endif

}  // namespace dcg

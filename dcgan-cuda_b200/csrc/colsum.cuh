// Column sums of a few hundred rows inside one block: shared by the column-sum launch and by the dense weight gradient, whose
// launch sums the same output gradient.
#pragma once

#include "common.cuh"

namespace dcg {

// The order in which the rows of a column are added: slabs of rows_per_slab rows; within a slab `lanes` lanes (a power of two)
// take every lanes-th row each, at most four, and a halving tree adds the lanes; then slab s goes to lane s % slab_lanes, and
// those are added in ascending order - first within groups of `group` slabs, if there are more, then the groups in the same
// way.  It follows from rows, columns and alignment alone, whoever computes it.
struct ColsumOrder {
    unsigned rows_per_slab, slabs, group;
    int lane_shift;    // lanes = 1 << lane_shift
    int slab_lanes;
};

// How a block computes it: 1 << tile_shift column groups (float4s or floats) at a time.
struct ColsumTile {
    ColsumOrder order;
    bool vec;
    unsigned groups;  // column groups
    int widest;       // tile_shift at most
    int tile_shift;
    unsigned tiles;   // column tiles
    size_t smem;      // bytes
};
// The order; false where it has more than `max_slabs` slabs or more than four rows per lane.
bool colsum_order(size_t rows, size_t cols, bool aligned, unsigned max_slabs, ColsumTile& t);
// The tile of a block of `threads` threads: the widest whose rows are all in flight at once and whose lanes are one warp's.
inline void colsum_fit(ColsumTile& t, int threads)
{
    const unsigned places = t.order.slabs << t.order.lane_shift;
    t.tile_shift = 0;
    while (t.tile_shift < t.widest && places << (t.tile_shift + 1) <= (unsigned)threads && t.order.lane_shift + t.tile_shift < 5) ++t.tile_shift;
    t.tiles = (t.groups + (1u << t.tile_shift) - 1) >> t.tile_shift;
    t.smem = ((size_t)places << t.tile_shift) * (t.vec ? 4 : 1) * sizeof(float);
}

#ifdef __CUDACC__
// Threads are [slab and lane][column group]: where a slab has few rows they run side by side, each with its rows in flight at
// once, instead of one slab after the other.  The lanes of a slab meet by shuffles where they are one warp's (a tile is chosen
// no wider than that allows, up to 32 lanes), in shared memory else.  All threads of the block take part; `threads` is a
// multiple of 32.
template <bool VEC>
__device__ __forceinline__ void colsum_tile_block(const float* __restrict__ a, float* __restrict__ out, const unsigned rows, const unsigned cols,
                                                  const ColsumOrder o, const int tile_shift, const unsigned block, const int threads, float* smem)
{
    constexpr int W = VEC ? 4 : 1;
    const int lanes = 1 << o.lane_shift, width_shift = tile_shift + (VEC ? 2 : 0), width = 1 << width_shift, tid = threadIdx.x;
    const int tx = tid & ((1 << tile_shift) - 1), step = threads >> tile_shift, places = (int)o.slabs << o.lane_shift;
    const unsigned group = (block << tile_shift) + tx, groups = cols / W;
    const bool one_warp = o.lane_shift + tile_shift <= 5;
    const int place_shift = one_warp ? 0 : o.lane_shift;   // places per slab in shared memory: [slab][place][column]
    for (int v0 = (tid & ~31) >> tile_shift; v0 < places; v0 += step) {   // whole warps
        const int v = v0 + ((tid & 31) >> tile_shift);
        const unsigned s = v >> o.lane_shift, r0 = s * o.rows_per_slab + (v & (lanes - 1)), r1 = min((s + 1) * o.rows_per_slab, rows);
        float acc[W];
#pragma unroll
        for (int q = 0; q < W; ++q) acc[q] = 0.f;
        if (group < groups && v < places) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const unsigned r = r0 + (i << o.lane_shift);
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
        if (one_warp) {   // h = 1 << hs lanes take over those h further on
            for (int hs = o.lane_shift - 1; hs >= 0; --hs)
#pragma unroll
                for (int q = 0; q < W; ++q) acc[q] += __shfl_down_sync(0xffffffffu, acc[q], 1 << (hs + tile_shift));
            if ((v & (lanes - 1)) != 0) continue;
        }
        if (v < places)
#pragma unroll
            for (int q = 0; q < W; ++q) smem[((one_warp ? (int)s : v) << width_shift) + tx * W + q] = acc[q];
    }
    __syncthreads();
    for (int hs = one_warp ? -1 : o.lane_shift - 1; hs >= 0; --hs) {
        for (int i = tid; i < (int)o.slabs << (hs + width_shift); i += threads) {
            const int u = i >> width_shift, place = (u >> hs << o.lane_shift) + (u & ((1 << hs) - 1));
            const int at = (place << width_shift) + (i & (width - 1));
            smem[at] += smem[at + (1 << (hs + width_shift))];
        }
        __syncthreads();
    }
    for (int i = tid; i < width; i += threads) {
        const unsigned c = (block << width_shift) + i;
        if (c >= cols) break;
        // n values over the lanes, each lane's and then the lanes in ascending order
        auto add = [&](unsigned n, auto value) {
            float r = 0.f;
            for (unsigned lane = 0; lane < min((unsigned)o.slab_lanes, n); ++lane) {
                float v = value(lane);
                for (unsigned s = lane + o.slab_lanes; s < n; s += o.slab_lanes) v += value(s);
                r = lane == 0 ? v : r + v;
            }
            return r;
        };
        auto slab_group = [&](unsigned g) {
            return add(min(o.group, o.slabs - g * o.group), [&](unsigned s) { return smem[((g * o.group + s) << (place_shift + width_shift)) + i]; });
        };
        out[c] = add((o.slabs + o.group - 1) / o.group, slab_group);
    }
}
#endif

}  // namespace dcg

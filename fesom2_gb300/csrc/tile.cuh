// tile.cuh -- tiles of columns: the wet levels of a few entities dealt to the threads of a block.
//
// A warp per column with its lanes over the levels leaves lanes idle wherever the column is not a
// multiple of 32 levels (47 layers: 32 + 15).  A tile numbers the wet levels of its entities one
// after another and gives thread i the items i, i + kTileThreads, ...: every warp but a tile's
// last is full, consecutive lanes still read consecutive levels, and a column's items are
// neighbours in any array over the items.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace fesom {

constexpr int kTileThreads = 128;
constexpr int kTileMax = 8;  // entities per tile

// tiles of nodes of the FP32 form, cut once per mesh: wet levels (= threads) and nodes of a tile
constexpr int kNodeTileLevels = 256, kNodeTileNodes = 32;

// the wet levels of a tile's entities as items 0 .. total-1: entity j holds the items
// pre[j] .. pre[j+1]-1, levels top[j], top[j] + 1, ...
struct Tile {
    int total;
    int pre[kTileMax + 1], top[kTileMax];
    // one warp, lane j < kTileMax with the level count of entity j (0 past the tile's end)
    __device__ __forceinline__ void fill(int lane, int first_level, int levels) {
        int s = lane < kTileMax ? levels : 0;
#pragma unroll
        for (int o = 1; o < kTileMax; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += v;
        }
        if (lane < kTileMax) {
            pre[lane + 1] = s;
            top[lane] = first_level;
            if (lane == 0) pre[0] = 0;
            if (lane == kTileMax - 1) total = s;
        }
    }
    __device__ __forceinline__ int find(int i) const {
        int j = i >= pre[4] ? 4 : 0;
        j += i >= pre[j + 2] ? 2 : 0;
        return j + (i >= pre[j + 1] ? 1 : 0);
    }
};

// entities per tile: 8, or 4 where 8 would leave less than eight blocks per SM (a mesh of 2.9k
// nodes: 4.8 blocks per SM instead of 2.4, so the SMs finish together); fewer where the tile's
// shared memory (`bytes` per entity) would pass 48 KB
static inline int tile_size(int n, size_t bytes) {
    int t = n >= 152 * 8 * kTileMax ? kTileMax : 4;
    while (t > 1 && t * bytes > 46 * 1024) t >>= 1;
    return t;
}

}  // namespace fesom

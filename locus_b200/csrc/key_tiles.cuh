// The key tiles that a tile of consecutive queries walks over, for the kernels whose tiles hold 64 keys: the first tile's first
// position and their number (the same in a walk and in the merge of its ranges).  With kept first tokens the tiles that hold
// them and lie in front of the window's first tile come first (kept_tiles of them, from position 0); tile number i of the
// item starts at tile_pos(i).
#pragma once
#include "mask.cuh"

#define KEY_TILE 64

__device__ __forceinline__ void item_tiles(int p0, int nq, int window, int chunk, int keep_first, int& first_tile, int& n_tiles,
                                           int& kept_tiles) {
    const int t_hi = p0 + nq - 1;
    const int t_lo = first_key(window, chunk, p0);
    first_tile = (t_lo / KEY_TILE) * KEY_TILE;
    kept_tiles = window > 0 ? min(first_tile / KEY_TILE, (min(keep_first, t_lo) + KEY_TILE - 1) / KEY_TILE) : 0;
    n_tiles = (t_hi - first_tile) / KEY_TILE + 1 + kept_tiles;
}
__device__ __forceinline__ int tile_pos(int i, int first_tile, int kept_tiles) {
    return i < kept_tiles ? i * KEY_TILE : first_tile + (i - kept_tiles) * KEY_TILE;
}

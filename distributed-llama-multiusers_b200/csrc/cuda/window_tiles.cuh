// Row tiles of windowed attention (tile_rows [n_tiles][rq], -1 where a tile has fewer rows): what the kernels that share a call's tiles
// (window_attention.cu, attention_prefill_tc.cu) must agree on, so that every tile has one owner.
#pragma once
#include <cuda_runtime.h>
#include "../../../include/dllama_b200.h"

__device__ __forceinline__ int window_tile_count(const int* tile_rows, int n_tiles, int rq, int u) {
    int n = 0;
    if (u < n_tiles)
        while (n < rq && tile_rows[(size_t)u * rq + n] >= 0) ++n;
    return n;
}

// tile e (ne rows) is full and tile e + 1 (no rows) continues its sequence: the tcgen05 kernel takes both in one run, however few rows
// the second has, unless e + 1 starts a group
__device__ __forceinline__ bool window_tiles_join(const DlWindowAttnArgs& a, const int* tile_rows, int rq, int e, int ne, int no) {
    if (ne != rq || no == 0) return false;
    const int me = tile_rows[(size_t)e * rq], mo = tile_rows[(size_t)(e + 1) * rq];
    return a.slot[me] == a.slot[mo] && a.pos[mo] == a.pos[me] + ne;
}

// Windows of the KV write kernels: which tokens a tile of 16 tokens writes (see kv_write_tiles.cuh, kv_write_staged.cuh).
// Plain arithmetic, so that it compiles on the host too.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define B200PA_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define B200PA_HOST_DEVICE inline
#endif

namespace b200pa {

// How far a tile with these first, ninth and last slots (below 0: none) is moved: up to the next 16-slot boundary
// of the cache, if the three are consecutive modulo 16.
B200PA_HOST_DEVICE int tile_shift(int64_t first, int64_t mid, int64_t last) {
  if (first < 0 || mid < 0 || last < 0) return 0;
  if (((mid - first) & 15) != 8 || ((last - first) & 15) != 15) return 0;
  return int((16 - (first & 15)) & 15);
}

// Rows lo .. hi - 1 of the 16 tokens from `tok` on.
struct TileWindow {
  int tok, lo, hi;
};

// The window of the tile at token t0 of n, moved by d: tokens of the next tile only if that one is moved as far.
B200PA_HOST_DEVICE TileWindow tile_window(int t0, int n, int d, int after) {
  const int rows = after == d ? 16 : 16 - d, left = n - t0 - d;
  return {t0 + d, 0, rows < left ? rows : left};
}

// What it gives up in front, empty where there is nothing or the tile before, moved as far, has it.
B200PA_HOST_DEVICE TileWindow tile_front_window(int t0, int d, int before) {
  return {t0 + d - 16, 16 - d, d > 0 && before != d ? 16 : 16 - d};
}

}  // namespace b200pa

// sw_resident2d.cuh -- launch parameters and shared-memory layout of the 2D
// time loops that stay on the chip (elastic2d_resident.cu).
#pragma once

#include <cstddef>

#include "sw_device.cuh"

namespace sw {

#define SW_RES_ORDER 4   // highest order with an on-chip loop
#define SW_RES_RECV 512  // receivers of one tile kept in its shared-memory table
#define SW_RES_MIN 8     // smallest tile side
#define SW_RES_FLOOR 540 // work of a tile (about its cells) below which less saves no time
#define SW_RES_STEPS 4   // fewest steps of a run that the on-chip loop takes

// One launch: the shot and its tx x tz tiles, one per block; tile (a, b) covers
// the rows between the cuts a and a+1 (res2_cut_x) and the columns between the
// cuts b and b+1 (res2_cut_z).  A tile's rim buffers (one per phase, `stride`
// 8-byte words each) start at word 2*tile*stride of the inbox; the tiles'
// agreement at the end of the run takes the word behind them.
template <typename T>
struct Res2 {
  P2<T> shot;
  int tx, tz, stride;
  int width;  // columns of a row block, 32 or 64 (every tile is at most that wide)
  size_t smem;
  uint64_t* inbox;
  int* err;
  int stop_tile;  // this tile behaves as if its last step's rims had not come (-1: none)
};

inline size_t res2_inbox_words(int tx, int tz, int stride) { return 2 * (size_t)tx * tz * stride + 1; }

// first column of tile t of tz: equal widths
__host__ __device__ __forceinline__ int res2_cut_z(int nz, int t, int tz) { return (int)((long long)t * nz / tz); }
// first row of tile t of tx: a row of the x slabs counts one and a half times
// (its CPML corrections), since the slowest tile sets the pace of all
__host__ __device__ __forceinline__ int res2_cut_x(int nx, int lo, int hi, int t, int tx) {
  const int mid = nx - lo - hi;
  const int w = (int)((long long)t * (3 * (lo + hi) + 2 * mid) / tx);
  if (w <= 3 * lo) return w / 3;
  if (w <= 3 * lo + 2 * mid) return lo + (w - 3 * lo) / 2;
  return lo + mid + (w - 3 * lo - 2 * mid) / 3;
}

__host__ __device__ __forceinline__ size_t res2_align16(size_t x) { return (x + 15) / 16 * 16; }

// shared memory of a tile of bx x bz cells in row blocks of `width` columns,
// with nsx slab rows and nsz slab columns: five fields with N-cell rims, seven
// material rows, the CPML memory variables and coefficient rows, the receiver
// table and a word per cell
__host__ __device__ __forceinline__ size_t res2_smem(int bx, int bz, int width, int nsx, int nsz, int N, int esz) {
  const size_t v = 5 * (size_t)(bx + 2 * N) * (width + 2 * N) + 7 * (size_t)bx * width + 4 * (size_t)nsx * bz +
                   4 * (size_t)bx * nsz + 8 * (size_t)(bx + bz);
  return res2_align16(v * esz) + 8 * SW_RES_RECV + 4 * (size_t)bx * width;
}

// Tiles for shot p on at most `blocks` SMs with `smem` bytes each: the split
// with the least work per tile (the fewest tiles among those of at most
// SW_RES_FLOOR), or false when none fits.  *words: 8-byte words
// of one rim buffer, *width: the row block's width.
template <typename T>
bool sw2r_tiles(const P2<T>& p, int N, int blocks, size_t smem, int* tx, int* tz, int* words, size_t* bytes,
                int* width);

// nsteps >= 1 steps of rs; aea: the free-surface hook precedes
// every step
template <typename T>
cudaError_t sw2r_run(const Res2<T>& rs, int scheme, int order, int it0, int nsteps, int aea, cudaStream_t st);

}  // namespace sw

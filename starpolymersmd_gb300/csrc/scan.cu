// Counting-sort support: exclusive prefix sum of the per-cell counts and the
// scatter that turns (cell, rank) keys into a cell-ordered permutation. This
// replaces MPC::sort's vector<vector<MPCParticle*>> push_back cell lists
// (star-polymers/lib/Hydrodynamics/MPC.cpp:201-237) with integer arithmetic.
//
// Scan: two launches over C cells: per-tile scan (count is re-zeroed for the
// next collision while it is read), then the totals of the tiles before are
// added; one launch of one CTA for few cells, and one between the two that
// scans the totals for very many. off[C] receives the total.
#include <stdint.h>

#include "launch.h"
#include "mpc_kernels.cuh"

namespace smpc {

constexpr int SCAN_NT = 256;
constexpr int SCAN_IPT = 8;
constexpr int SCAN_TILE = SCAN_NT * SCAN_IPT;

// One tile of SCAN_TILE cells per CTA. Warp w owns the tile's w-th run of
// 32 * SCAN_IPT consecutive cells, read as SCAN_IPT rows of 32 (every load and
// store of a warp is one contiguous 128-byte row); each row is a warp scan
// carried into the next, then the warps' totals give each warp's base.
// Offsets are within the tile; k_scan_add adds the tiles before. A scan of one
// tile is complete (one launch).
template <int NT, int IPT>
__global__ void __launch_bounds__(NT) k_scan_tiles(uint32_t* __restrict__ count,
                                                   uint32_t* __restrict__ off,
                                                   uint32_t* __restrict__ tile_sum, int n) {
  __shared__ uint32_t warp_tot[NT / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int seg = blockIdx.x * (NT * IPT) + w * (32 * IPT);
  uint32_t c[IPT], pre[IPT];
#pragma unroll
  for (int k = 0; k < IPT; ++k) {
    const int i = seg + 32 * k + lane;
    c[k] = i < n ? count[i] : 0u;
  }
#pragma unroll
  for (int k = 0; k < IPT; ++k) {
    const int i = seg + 32 * k + lane;
    if (i < n) count[i] = 0u;  // re-zeroed for the next collision
  }
  uint32_t carry = 0;
#pragma unroll
  for (int k = 0; k < IPT; ++k) {
    uint32_t x = c[k];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
      if (lane >= o) x += y;
    }
    pre[k] = carry + x - c[k];
    carry += __shfl_sync(0xFFFFFFFFu, x, 31);
  }
  if (lane == 0) warp_tot[w] = carry;
  __syncthreads();
  uint32_t wbase = 0, total = 0;
#pragma unroll
  for (int q = 0; q < NT / 32; ++q) {
    const uint32_t t = warp_tot[q];
    if (q < w) wbase += t;
    total += t;
  }
#pragma unroll
  for (int k = 0; k < IPT; ++k) {
    const int i = seg + 32 * k + lane;
    if (i < n) off[i] = wbase + pre[k];
  }
  if (threadIdx.x == 0) {
    tile_sum[blockIdx.x] = total;
    if (gridDim.x == 1) off[n] = total;
  }
}

// Adds the totals of the tiles before to a tile's offsets; every CTA sums them
// for itself, beside its loads of the offsets, instead of waiting for a launch
// that scans them. (A single launch with decoupled look-back, each tile polling
// its predecessors' totals, took 9.3 us for 62 tiles and 67 for 3,907; the two
// launches take 6.4 and 24, three with one for the totals took 9 and 28; for
// very many tiles see SCAN_MANY.)
// SCANNED: tile_sum holds the sums before each tile already (k_scan_totals).
template <bool SCANNED>
__global__ void __launch_bounds__(SCAN_NT) k_scan_add(uint32_t* __restrict__ off,
                                                      const uint32_t* __restrict__ tile_sum,
                                                      int n) {
  __shared__ uint32_t warp_tot[SCAN_NT / 32];
  const int tile = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int base = tile * SCAN_TILE + threadIdx.x;
  uint32_t v[SCAN_IPT];
#pragma unroll
  for (int u = 0; u < SCAN_IPT; ++u) {
    const int i = base + u * SCAN_NT;
    v[u] = i < n ? off[i] : 0u;
  }
  uint32_t before = 0;
  if (SCANNED) {
    before = tile_sum[tile];
  } else {
#pragma unroll 4
    for (int t = threadIdx.x; t < tile; t += SCAN_NT) before += tile_sum[t];
    before = __reduce_add_sync(0xFFFFFFFFu, before);
    if (lane == 0) warp_tot[w] = before;
    __syncthreads();
    before = 0;
#pragma unroll
    for (int q = 0; q < SCAN_NT / 32; ++q) before += warp_tot[q];
  }
#pragma unroll
  for (int u = 0; u < SCAN_IPT; ++u) {
    const int i = base + u * SCAN_NT;
    if (i < n) off[i] = v[u] + before;
  }
  if (!SCANNED && tile == static_cast<int>(gridDim.x) - 1 && threadIdx.x == 0)
    off[n] = before + tile_sum[tile];
}

// The tiles' totals, scanned in place by one CTA; off[n] receives their sum.
constexpr int SCAN_TOT_NT = 1024, SCAN_TOT_IPT = 8;
__global__ void __launch_bounds__(SCAN_TOT_NT) k_scan_totals(uint32_t* __restrict__ tile_sum,
                                                             int tiles, uint32_t* __restrict__ off,
                                                             int n) {
  __shared__ uint32_t warp_tot[SCAN_TOT_NT / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t carry = 0;
  for (int base = 0; base < tiles; base += SCAN_TOT_NT * SCAN_TOT_IPT) {
    const int first = base + threadIdx.x * SCAN_TOT_IPT;
    uint32_t c[SCAN_TOT_IPT], own = 0;
#pragma unroll
    for (int k = 0; k < SCAN_TOT_IPT; ++k) {
      c[k] = first + k < tiles ? tile_sum[first + k] : 0u;
      own += c[k];
    }
    uint32_t x = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[w] = x;
    __syncthreads();
    uint32_t run = carry + x - own;
#pragma unroll
    for (int q = 0; q < SCAN_TOT_NT / 32; ++q) {
      const uint32_t t = warp_tot[q];
      if (q < w) run += t;
      carry += t;
    }
#pragma unroll
    for (int k = 0; k < SCAN_TOT_IPT; ++k) {
      if (first + k < tiles) tile_sum[first + k] = run;
      run += c[k];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) off[n] = carry;
}

// perm[off[cell] + rank] = source. Each thread takes PERM_U entries a block
// apart and issues all key loads, then all offset gathers, then the stores,
// so PERM_U independent gather chains are in flight per thread. A position
// past the last entry (counts that do not match the keys; never expected) is
// reported in the error word, not written.
constexpr int PERM_NT = 256;
constexpr int PERM_U = 4;
__global__ void __launch_bounds__(PERM_NT) k_build_perm(const uint2* __restrict__ keys, int n_slots,
                                                        const uint2* __restrict__ mkey, int n_mono,
                                                        const uint32_t* __restrict__ off,
                                                        uint32_t* __restrict__ perm,
                                                        ErrorState* err) {
  const int n = n_slots + n_mono;
  const int base = blockIdx.x * (PERM_NT * PERM_U) + threadIdx.x;
  uint2 k[PERM_U];
#pragma unroll
  for (int u = 0; u < PERM_U; ++u) {
    const int i = base + u * PERM_NT;
    k[u] = make_uint2(KEY_NONE, 0u);
    if (i < n_slots)
      k[u] = keys[i];
    else if (i < n)
      k[u] = mkey[i - n_slots];
  }
  uint32_t o[PERM_U];
#pragma unroll
  for (int u = 0; u < PERM_U; ++u) o[u] = k[u].x != KEY_NONE ? off[k[u].x] : 0u;
#pragma unroll
  for (int u = 0; u < PERM_U; ++u) {
    const int i = base + u * PERM_NT;
    if (k[u].x == KEY_NONE) continue;
    const uint32_t pos = o[u] + k[u].y;
    if (pos < static_cast<uint32_t>(n))
      perm[pos] = i < n_slots ? static_cast<uint32_t>(i) : (MONO_BIT | static_cast<uint32_t>(i - n_slots));
    else
      raise_error(err, ERR_KEY_MISMATCH, pos, k[u].x);
  }
}

// The same scatter from packed solvent keys (local cell << 16 | rank, written
// by the packed binning): one block per binning tile of slots, whose replica
// gives the cell base; the monomers' (global cell, rank) keys in the blocks
// after the tiles.
__global__ void __launch_bounds__(PERM_NT) k_build_perm_packed(
    const Tile* tiles, int n_tiles, const RepInfo* reps, const uint32_t* __restrict__ keys,
    int n_slots, const uint2* __restrict__ mkey, int n_mono, const uint32_t* __restrict__ off,
    uint32_t* __restrict__ perm, ErrorState* err) {
  const uint32_t n = static_cast<uint32_t>(n_slots + n_mono);
  if (static_cast<int>(blockIdx.x) < n_tiles) {
    const Tile t = tiles[blockIdx.x];
    const uint32_t cbase = static_cast<uint32_t>(reps[t.rep].cell_base);
    for (int base = t.begin + static_cast<int>(threadIdx.x); base < t.end;
         base += PERM_NT * PERM_U) {
      uint32_t k[PERM_U], o[PERM_U];
#pragma unroll
      for (int u = 0; u < PERM_U; ++u) {
        const int i = base + u * PERM_NT;
        k[u] = i < t.end ? keys[i] : KEY_NONE;
      }
#pragma unroll
      for (int u = 0; u < PERM_U; ++u) o[u] = k[u] != KEY_NONE ? off[cbase + (k[u] >> 16)] : 0u;
#pragma unroll
      for (int u = 0; u < PERM_U; ++u) {
        if (k[u] == KEY_NONE) continue;
        const uint32_t pos = o[u] + (k[u] & 0xFFFFu);
        if (pos < n)
          perm[pos] = static_cast<uint32_t>(base + u * PERM_NT);
        else
          raise_error(err, ERR_KEY_MISMATCH, pos, k[u]);
      }
    }
    return;
  }
  const int base = (static_cast<int>(blockIdx.x) - n_tiles) * (PERM_NT * PERM_U) +
                   static_cast<int>(threadIdx.x);
#pragma unroll
  for (int u = 0; u < PERM_U; ++u) {
    const int i = base + u * PERM_NT;
    if (i >= n_mono) continue;
    const uint2 k = mkey[i];
    if (k.x == KEY_NONE) continue;
    const uint32_t pos = off[k.x] + k.y;
    if (pos < n)
      perm[pos] = MONO_BIT | static_cast<uint32_t>(i);
    else
      raise_error(err, ERR_KEY_MISMATCH, pos, k.x);
  }
}

// Up to this many cells one CTA scans them all: 5.1 us for 8,000 cells, against
// 6.5 and a launch more in two (8.5 in three, with one for the totals); with
// four times as many cells per thread it took 12 us for 29,791.
constexpr int SCAN_ONE_NT = 1024, SCAN_ONE_IPT = 8;
constexpr int SCAN_ONE = SCAN_ONE_NT * SCAN_ONE_IPT;
// Above this many tiles (67 M cells) a third launch scans their totals: every
// CTA's own sum over the tiles before it grows with their number. Two launches
// against three: 56 and 61 us for 8,192 tiles, 214 and 214 for 31,250, 370 and
// 301 for 44,494, 668 and 410 for 61,035.
constexpr int SCAN_MANY = 32768;
int scan_tile_count(int n_cells) { return (n_cells + SCAN_TILE - 1) / SCAN_TILE; }

void launch_scan(uint32_t* count, uint32_t* off, uint32_t* tile_sum, int n_cells,
                 cudaStream_t st) {
  if (n_cells <= SCAN_ONE) {
    k_scan_tiles<SCAN_ONE_NT, SCAN_ONE_IPT><<<1, SCAN_ONE_NT, 0, st>>>(count, off, tile_sum,
                                                                       n_cells);
    return;
  }
  const int tiles = scan_tile_count(n_cells);
  k_scan_tiles<SCAN_NT, SCAN_IPT><<<tiles, SCAN_NT, 0, st>>>(count, off, tile_sum, n_cells);
  if (tiles > SCAN_MANY) {
    k_scan_totals<<<1, SCAN_TOT_NT, 0, st>>>(tile_sum, tiles, off, n_cells);
    k_scan_add<true><<<tiles, SCAN_NT, 0, st>>>(off, tile_sum, n_cells);
  } else {
    k_scan_add<false><<<tiles, SCAN_NT, 0, st>>>(off, tile_sum, n_cells);
  }
}

void launch_build_perm_packed(const Tile* tiles, int n_tiles, const RepInfo* reps,
                              const uint32_t* keys, int n_slots, const uint2* mkey, int n_mono,
                              const uint32_t* off, uint32_t* perm, ErrorState* err,
                              cudaStream_t st) {
  const int mono_blocks = (n_mono + PERM_NT * PERM_U - 1) / (PERM_NT * PERM_U);
  if (n_tiles + mono_blocks == 0) return;
  k_build_perm_packed<<<n_tiles + mono_blocks, PERM_NT, 0, st>>>(tiles, n_tiles, reps, keys,
                                                                 n_slots, mkey, n_mono, off, perm,
                                                                 err);
}

void launch_build_perm(const uint2* keys, int n_slots, const uint2* mkey, int n_mono,
                       const uint32_t* off, uint32_t* perm, ErrorState* err, cudaStream_t st) {
  const int n = n_slots + n_mono;
  if (n == 0) return;
  k_build_perm<<<(n + PERM_NT * PERM_U - 1) / (PERM_NT * PERM_U), PERM_NT, 0, st>>>(
      keys, n_slots, mkey, n_mono, off, perm, err);
}

}  // namespace smpc

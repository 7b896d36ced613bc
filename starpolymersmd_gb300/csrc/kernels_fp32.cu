// FP32 fast-path instantiation: float4 state, int64 fixed-point cell sums.
#define SMPC_REAL float
#define SMPC_FAST_F32 1
#define SMPC_COLLIDE_NT 256
#define SMPC_COLLIDE_CT 128
#define SMPC_COLLIDE_CAP 1408
#define SMPC_COLLIDE_BLOCKS 3
#define SMPC_BIN_NT 256
#define SMPC_MD_NT 1024
#define SMPC_MD_MPT 1
#include <cmath>

#include "kernels_impl.cuh"

namespace smpc {
// Variant tables (index 0 is the default shape).
int bin_variant_count() { return 4; }
int collide_variant_count() { return 12; }  // indices accepted; one shape
int collide_shape_count() { return 1; }
int md_variant_count() { return 5; }
// Cells per collide tile of a box with `density` particles per cell, in a
// context of total_cells: as many as the tile has lane pairs for (32) and
// staging room for, the mean and 3.3 standard deviations of a Poisson count
// (30 cells at 10 per cell: a tile past its staging room reads the rest from
// global memory again; 154 us against 156 with 32 cells on 10 M particles),
// but no more than gives every SM four tiles (13 in 20^3 cells: 10.3 us
// against 15.3 with 32; 8 and fewer leave too many lanes without a cell).
int collide_tile_cells(double density, long long total_cells) {
  int ct = COL_CT;
  while (ct > 4 && ct * density + 3.3 * std::sqrt(ct * density) > COL_CAP) --ct;
  return std::min(ct, std::max(8, static_cast<int>(std::min(total_cells / (152 * 4), 64ll))));
}
const char* bin_variant_name(int v) {
  static const char* n[] = {"256t x4", "256t x2", "256t x8", "128t x8"};
  return v >= 0 && v < 4 ? n[v] : "?";
}
const char* collide_variant_name(int) { return "64t 32c cap360 cp.async"; }
int pmd_variant_count() { return 4; }
int pmd_variant_lanes(int v) {
  static const int lanes[] = {8, 4, 16, 8};
  return v >= 0 && v < 4 ? lanes[v] : 8;
}
int pmd_variant_list_blocks_per_sm(int v) { return v == 3 ? 8 : 4; }
const char* pmd_variant_name(int v) {
  static const char* n[] = {"8 lanes/bead, lists 4 blocks/SM", "4 lanes/bead, lists 4 blocks/SM",
                            "16 lanes/bead, lists 4 blocks/SM", "8 lanes/bead, lists 8 blocks/SM"};
  return v >= 0 && v < 4 ? n[v] : "?";
}
const char* md_variant_name(int v) {
  static const char* n[] = {"1024t 1/thread", "512t 2/thread", "1024t lanes/bead, largest first",
                            "1024t big + 512t small side by side, lanes/bead",
                            "cluster of SMs per replica (few replicas; else 1024t 1/thread)"};
  return v >= 0 && v < 5 ? n[v] : "?";
}
}  // namespace smpc

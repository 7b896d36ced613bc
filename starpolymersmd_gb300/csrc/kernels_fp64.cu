// FP64 reference-parity instantiation. Built with -fmad=false so every
// multiply and add rounds separately, in the reference's order. Fused operations
// are written out in the collision itself (cell sums, rotation with the
// thermostat's factor), the gamma variate and the kinetic stress; the cluster MD
// adds a bead's even and odd force terms apart.
#define SMPC_REAL double
#define SMPC_FAST_F32 0
#define SMPC_COLLIDE_NT 128
#define SMPC_COLLIDE_CT 64
#define SMPC_COLLIDE_CAP 768
#define SMPC_COLLIDE_BLOCKS 3
#define SMPC_BIN_NT 256
#define SMPC_MD_NT 256
#define SMPC_MD_MPT 4
#include "kernels_impl.cuh"

namespace smpc {
// Solvent slots per binning tile (one CTA): FP64 blocks hold two records per
// thread in flight (k_fluid_bin), FP32 blocks four. At most two (four) rounds of
// these, and down to one so that a small box still gives every SM several CTAs
// to hide the atomics' round trips: FP32, 80,000 particles: 79 tiles of 1,024
// bin in 6.4 us, 20 of 4,096 in 15; 1.5 M: 742 of 2,048 in 18.0, 371 of 4,096 in
// 19.4. FP64, 640,000 particles: tiles of 512 in 49 us, of 1,024 and 2,048 in 54;
// 1.25 M: 83, 83, 87.
int fluid_slots_per_tile(bool fp64, long long slots) {
  int n = fp64 ? 1024 : 4096;
  const int least = fp64 ? 512 : 1024;
  while (n > least && slots < n * (fp64 ? 8ll : 4ll) * 152) n /= 2;
  return n;
}
int temperature_cells_per_tile() { return 512; }
int md_max_monomers() { return SMPC_MD_NT * SMPC_MD_MPT; }
// Runs so long that the SMs keep 1,024 threads each, up to 16 slots: 5,120
// slots 44 us the call with runs of one and 70 with 16, 1.25 M 121 to 127 with 4
// or 8 and 125 to 133 with 16, 10 M 593 to 626 with 16 and 888 with one.
// Copies of the bins where 300 or more particles meet in one (bins counts three
// doubles for each, x and y): 80,000 particles and 2,001 bins per axis take 48 us
// without copies and 62 with 128 of them, 201 bins 61 and 52; 1.25 M particles and
// 5,001 bins 129 and 154, 501 bins 162 and 133. No more copies than blocks, and
// none past 65,536 doubles.
ProfilePlan profile_plan(int slots, size_t bins) {
  int run = 1;
  while (run < 16 && slots >= 2 * run * 152 * 1024) run *= 2;
  const int blocks = (slots + PROF_NT * run - 1) / (PROF_NT * run);
  const bool copies = bins <= 65536 && static_cast<size_t>(slots) >= 50 * bins;
  return {copies ? std::max(1, std::min(128, blocks)) : 1, run};
}
// A block for every eight beads (one round of its 256 threads), or fewer where all
// replicas' blocks would be more than eight per SM. With as many for each replica
// as for the largest, 64 stars of 31 to 721 beads took 178 us the call, now 131,
// and 200 of 10 beads beside a box of 6,420 took 1,908, now 132.
int stress_blocks(int n_mono, long long total_mono) {
  constexpr long long beads = ANA_NT / STRESS_LANES, most = 152 * 8;
  const long long need = (n_mono + beads - 1) / beads, all = (total_mono + beads - 1) / beads;
  return static_cast<int>(std::max(1ll, all <= most ? need : need * most / all));
}
int pmd_block_count(int n_beads) { return (n_beads + PMD_NT - 1) / PMD_NT; }
}  // namespace smpc

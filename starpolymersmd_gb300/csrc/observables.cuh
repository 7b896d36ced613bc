// Output-step observables on the device, FP64 (star-polymers.cpp:466-483):
//   k_mol_observables  per replica: radius of gyration and gyration tensor
//                      (Box::calculate_gyration_tensor, Box.cpp:330-353),
//                      rotation frequency (Box::calculate_rotation_frequency,
//                      Box.cpp:355-379), kinetic energy and temperature
//                      (Box::calculate_ekin / print_Ekin_and_Temperature,
//                      Box.cpp:288-294, 635-646), all in each molecule's
//                      centre-of-mass frame (Box::center_of_mass_reference_frame,
//                      Box.cpp:81-102);
//   k_velocity_profile VelocityX (Velocity_x.h:76-100): solvent velocity
//                      relative to molecule 0's centre-of-mass velocity, binned
//                      by the Lees-Edwards-wrapped position relative to its
//                      centre of mass, along x and along y.
// Centres of mass are summed by one thread in monomer order, like the
// reference, so every position relative to them is the reference's to the
// last bit; the tensor, momentum and energy sums are block reductions.
#pragma once
#include <stdint.h>

#include <type_traits>

#include "mpc_kernels.cuh"
#include "smpc_device.cuh"

namespace smpc {

constexpr int OBS_PER_REP = 16;
constexpr int UNWRAP_NT = 256;  // threads (and beads per chunk) of k_unwrap_molecules

// Centre of molecule [b, e), unweighted mean position and velocity, summed in
// monomer order like the reference. The block stages the monomers in shared
// memory, then six lanes add one component each: one thread that loaded and
// added everything itself waited for memory at every monomer (185 us for 401
// of them). c (shared) is valid after the caller's barrier.
constexpr int CENTRE_CHUNK = 256;
template <typename R, int NT>
__device__ __forceinline__ void molecule_centre(const R* mpos, const R* mvel, int b, int e,
                                                R (*stage)[CENTRE_CHUNK], double* c) {
  double s = 0.0;
  for (int base = b; base < e; base += CENTRE_CHUNK) {
    const int n = min(CENTRE_CHUNK, e - base);
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += NT) {
      const R4<R> p = ld4_rw(mpos, base + i), v = ld4_rw(mvel, base + i);
      stage[0][i] = p.x;
      stage[1][i] = p.y;
      stage[2][i] = p.z;
      stage[3][i] = v.x;
      stage[4][i] = v.y;
      stage[5][i] = v.z;
    }
    __syncthreads();
    if (threadIdx.x < 6) {
#pragma unroll 8
      for (int i = 0; i < n; ++i) s += to_d(stage[threadIdx.x][i]);
    }
  }
  if (threadIdx.x < 6) c[threadIdx.x] = s / static_cast<double>(e - b);
}

// x = A^-1 b for a symmetric positive-definite 3x3 A (LDL^T, no pivoting)
__device__ __forceinline__ void solve_sym3(const double A[3][3], const double b[3], double x[3]) {
  double L10 = 0, L20 = 0, L21 = 0, D0, D1, D2;
  D0 = A[0][0];
  L10 = A[1][0] / D0;
  L20 = A[2][0] / D0;
  D1 = A[1][1] - L10 * L10 * D0;
  L21 = (A[2][1] - L20 * L10 * D0) / D1;
  D2 = A[2][2] - L20 * L20 * D0 - L21 * L21 * D1;
  const double y0 = b[0];
  const double y1 = b[1] - L10 * y0;
  const double y2 = b[2] - L20 * y0 - L21 * y1;
  x[2] = y2 / D2;
  x[1] = y1 / D1 - L21 * x[2];
  x[0] = y0 / D0 - L10 * x[1] - L20 * x[2];
}

template <int NT>
__device__ __forceinline__ double block_sum(double v, double* s_red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < NT / 32; ++w) t += s_red[w];
  return t;  // valid in thread 0
}

// K block sums at once into out[k] (shared; valid in every thread on return),
// in a fixed order: every thread's values through shared memory, then warp w
// sums values w, w + NT / 32, ...: NT / 32 partials per lane and one butterfly
// per value (a butterfly per value in every warp took NT / 32 times the FP64
// instructions). s_red holds K * NT doubles.
template <int NT, int K>
__device__ __forceinline__ void block_sum_n(double (&v)[K], double* s_red, double* out) {
#pragma unroll
  for (int k = 0; k < K; ++k) s_red[k * NT + threadIdx.x] = v[k];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int k = threadIdx.x >> 5; k < K; k += NT / 32) {
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < NT / 32; ++w) t += s_red[k * NT + 32 * w + lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, o);
    if (lane == 0) out[k] = t;
  }
  __syncthreads();
}

// FP32 contexts: the same centre as a block reduction (7 us for 401 monomers,
// with the kernel's launch).
template <int NT>
__device__ __forceinline__ void molecule_centre_f32(const float* mpos, const float* mvel, int b,
                                                    int e, double* s_red, double* s_tot,
                                                    double* c) {
  double t[6] = {0, 0, 0, 0, 0, 0};
  for (int i = b + threadIdx.x; i < e; i += NT) {
    const R4<float> p = ld4_rw(mpos, i), v = ld4_rw(mvel, i);
    t[0] += to_d(p.x);
    t[1] += to_d(p.y);
    t[2] += to_d(p.z);
    t[3] += to_d(v.x);
    t[4] += to_d(v.y);
    t[5] += to_d(v.z);
  }
  block_sum_n<NT, 6>(t, s_red, s_tot);
  if (threadIdx.x < 6) c[threadIdx.x] = s_tot[threadIdx.x] / static_cast<double>(e - b);
}

// One CTA per molecule; mols[m] = global monomer range [x, y). mol_out[16 m
// + ...]: R_g of the molecule, G (row-major, 9), rotation frequency (3),
// kinetic energy, monomers. FP64 sums the centre in monomer order (the
// reference's order, so the relative positions are the reference's to the
// last bit); FP32 sums it as a block reduction.
template <typename R, int NT>
__global__ void __launch_bounds__(NT) k_mol_observables(const int2* mols, const R* mpos,
                                                        const R* mvel, double* mol_out) {
  __shared__ double s_c[6];
  __shared__ double s_red[10 * NT];
  __shared__ double s_tot[10];
  const int2 mb = mols[blockIdx.x];
  const int n = mb.y - mb.x;
  if constexpr (std::is_same<R, double>::value) {
    __shared__ R s_stage[6][CENTRE_CHUNK];
    molecule_centre<R, NT>(mpos, mvel, mb.x, mb.y, s_stage, s_c);
  } else {
    molecule_centre_f32<NT>(mpos, mvel, mb.x, mb.y, s_red, s_tot, s_c);
  }
  __syncthreads();
  // S = sum r r^T (6), angular momentum (3), sum m |u|^2
  double acc[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (int i = mb.x + threadIdx.x; i < mb.y; i += NT) {
    const R4<R> p = ld4_rw(mpos, i), v = ld4_rw(mvel, i);
    const double x0 = static_cast<double>(p.x) - s_c[0], x1 = static_cast<double>(p.y) - s_c[1],
                 x2 = static_cast<double>(p.z) - s_c[2];
    const double u0 = static_cast<double>(v.x) - s_c[3], u1 = static_cast<double>(v.y) - s_c[4],
                 u2 = static_cast<double>(v.z) - s_c[5];
    acc[0] += x0 * x0;
    acc[1] += x0 * x1;
    acc[2] += x0 * x2;
    acc[3] += x1 * x1;
    acc[4] += x1 * x2;
    acc[5] += x2 * x2;
    acc[6] += x1 * u2 - x2 * u1;
    acc[7] += x2 * u0 - x0 * u2;
    acc[8] += x0 * u1 - x1 * u0;
    acc[9] += static_cast<double>(p.w) * ((u0 * u0 + u1 * u1) + u2 * u2);
  }
  block_sum_n<NT, 10>(acc, s_red, s_tot);
  if (threadIdx.x != 0) return;
  double tot[10];
  for (int k = 0; k < 10; ++k) tot[k] = s_tot[k];
  double* o = mol_out + static_cast<size_t>(OBS_PER_REP) * blockIdx.x;
  for (int k = 0; k < OBS_PER_REP; ++k) o[k] = 0.0;
  if (n <= 0) return;
  const double dn = static_cast<double>(n);
  double g[9];
  if (std::is_same<R, double>::value) {  // the reference's divisions (Box.cpp:330-379)
    const double gg[9] = {tot[0] / dn, tot[1] / dn, tot[2] / dn, tot[1] / dn, tot[3] / dn,
                          tot[4] / dn, tot[2] / dn, tot[4] / dn, tot[5] / dn};
    for (int k = 0; k < 9; ++k) g[k] = gg[k];
  } else {  // FP32 path: one division
    const double inv = 1.0 / dn;
    const double gg[9] = {tot[0] * inv, tot[1] * inv, tot[2] * inv, tot[1] * inv, tot[3] * inv,
                          tot[4] * inv, tot[2] * inv, tot[4] * inv, tot[5] * inv};
    for (int k = 0; k < 9; ++k) g[k] = gg[k];
  }
  for (int k = 0; k < 9; ++k) o[1 + k] = g[k];
  o[0] = sqrt(g[0] + g[4] + g[8]);
  const double tr = tot[0] + tot[3] + tot[5];
  const double I[3][3] = {{tr - tot[0], -tot[1], -tot[2]},
                          {-tot[1], tr - tot[3], -tot[4]},
                          {-tot[2], -tot[4], tr - tot[5]}};
  const double Lm[3] = {tot[6], tot[7], tot[8]};
  double om[3];
  solve_sym3(I, Lm, om);
  for (int k = 0; k < 3; ++k) o[10 + k] = om[k];
  o[13] = tot[9] * 0.5;
  o[14] = dn;
}

// One warp per replica: means over its molecules. out[16 r
// + ...]: mean R_g, mean G (row-major, 9), mean rotation frequency (3),
// kinetic energy, temperature 2 E / (3 (N - 1)), molecules.
template <typename R>  // R: the precision of the instantiating unit (one copy per unit)
__global__ void k_obs_reduce(const int2* rep_mols, const double* mol_out, int n_rep, double* out) {
  // one warp per replica: lane l sums molecules l, l + 32, ... in order, then
  // a fixed xor butterfly joins the lanes; lane 0 writes (a replica of one
  // molecule gets its values unchanged)
  constexpr unsigned FULL = 0xFFFFFFFFu;
  const int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (r >= n_rep) return;  // whole warps
  const int2 rm = rep_mols[r];
  double acc[14];  // R_g, G (9), rotation frequency (3), kinetic energy
#pragma unroll
  for (int k = 0; k < 14; ++k) acc[k] = 0.0;
  long long n_total = 0;
  for (int m = rm.x + lane; m < rm.x + rm.y; m += 32) {
    const double* o = mol_out + static_cast<size_t>(OBS_PER_REP) * m;
    double v[15];
#pragma unroll
    for (int k = 0; k < 15; ++k) v[k] = o[k];
    if (v[14] <= 0.0) continue;
#pragma unroll
    for (int k = 0; k < 14; ++k) acc[k] += v[k];
    n_total += static_cast<long long>(v[14]);
  }
  // (one molecule: the other lanes' zeros change nothing)
  for (int off = rm.y > 1 ? 16 : 0; off > 0; off >>= 1) {
#pragma unroll
    for (int k = 0; k < 14; ++k) acc[k] += __shfl_xor_sync(FULL, acc[k], off);
    n_total += __shfl_xor_sync(FULL, n_total, off);
  }
  if (lane != 0) return;
  const double nm = rm.y > 0 ? static_cast<double>(rm.y) : 1.0;
  double* o = out + static_cast<size_t>(OBS_PER_REP) * r;
  if (std::is_same<R, double>::value) {
    // the reference's divisions by Molecules.size() (Box.cpp:350-351, 378)
    o[0] = acc[0] / nm;
    for (int k = 0; k < 9; ++k) o[1 + k] = acc[1 + k] / nm;
    for (int k = 0; k < 3; ++k) o[10 + k] = acc[10 + k] / nm;
  } else {
    // FP32 path: one division (FP64 divisions are slow on this part); exact
    // for one molecule
    const double inv = 1.0 / nm;
    o[0] = acc[0] * inv;
    for (int k = 0; k < 9; ++k) o[1 + k] = acc[1 + k] * inv;
    for (int k = 0; k < 3; ++k) o[10 + k] = acc[10 + k] * inv;
  }
  o[13] = acc[13];
  o[14] = n_total > 1 ? acc[13] * 2. / (3. * static_cast<double>(n_total - 1)) : 0.0;
  o[15] = static_cast<double>(rm.y);
}

// Molecules of periodic boxes made whole for the observables: bead i is placed
// at the Lees-Edwards minimum image (MPC.cpp:456-465, current delrx) next to
// its lowest-indexed bonded partner in the molecule, which comes earlier and is
// already placed, or next to the molecule's first bead when it has none. Its
// v_x gets the shear velocity of the image it moved to (MPC.cpp:428).
// k_copy_monomers copies every monomer first; k_unwrap_molecules then runs one
// CTA per molecule of a periodic box over chunks of UNWRAP_NT beads: when
// every bead of a chunk has its partner either before the chunk (placed) or
// right before itself (stars and chains numbered outward from the core), the
// chunk is one segmented prefix sum of the bond vectors (warp scans joined in
// warp order); otherwise thread 0 walks it.
template <typename R>
__global__ void k_copy_monomers(int n, const R* mpos, const R* mvel, R* upos, R* uvel) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    st4(upos, i, ld4_rw(mpos, i));
    st4(uvel, i, ld4_rw(mvel, i));
  }
}

// Lees-Edwards minimum image of a bond vector. The image counts come from
// products with 1 / L: a bond is far shorter than half the box, so d / L is
// never near a half-integer and the count is the one the division gives.
__device__ __forceinline__ void unwrap_bond(const double L[3], const double invL[3], double delrx,
                                            double& d0, double& d1, double& d2) {
  const double cy = round(d1 * invL[1]);
  d0 -= L[0] * round(d0 * invL[0]);
  d0 -= cy * delrx;
  d0 -= L[0] * round(d0 * invL[0]);
  d1 -= L[1] * cy;
  d2 -= L[2] * round(d2 * invL[2]);
}

template <typename R>
__global__ void __launch_bounds__(UNWRAP_NT)
    k_unwrap_molecules(const RepInfo* reps, const RepDyn* dyn, const int2* mols,
                       const int* mol_rep, int n_mols, const int* bond_start, const int2* bonds,
                       const R* mpos, const R* mvel, R* upos, R* uvel) {
  constexpr unsigned FULL = 0xFFFFFFFFu;
  constexpr int NW = UNWRAP_NT / 32;
  __shared__ double s_wsum[3][NW];  // per warp: the scan value of its last lane
  __shared__ int s_whead[NW];       // per warp: it holds a segment head
  __shared__ double s_carry[3][NW];  // per warp: what its leading (headless) lanes add
  __shared__ int s_walk;            // the chunk needs the one-by-one walk
  __shared__ int s_p[UNWRAP_NT];
  __shared__ double s_d[3][UNWRAP_NT];
  const int m = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const RepInfo& ri = reps[mol_rep[m]];
  if (!(ri.flags & REP_PERIODIC_MD)) return;  // whole block
  const double L[3] = {static_cast<double>(ri.L[0]), static_cast<double>(ri.L[1]),
                       static_cast<double>(ri.L[2])};
  const double invL[3] = {1.0 / L[0], 1.0 / L[1], 1.0 / L[2]};
  const double delrx = dyn[mol_rep[m]].delrx;
  const double sLy = ri.shear * L[1];
  const int2 mb = mols[m];
  for (int c0 = mb.x + 1; c0 < mb.y; c0 += UNWRAP_NT) {
    const int i = c0 + tid;
    const bool active = i < mb.y;
    int p = -1;
    double d0 = 0, d1 = 0, d2 = 0, xy = 0, uy = 0;
    if (tid == 0) s_walk = 0;
    if (active) {
      for (int e = bond_start[i]; e < bond_start[i + 1]; ++e) {
        const int j = bonds[e].x;
        if (j >= mb.x && j < i && (p < 0 || j < p)) p = j;
      }
      if (p < 0) p = mb.x;
      const R4<R> x = ld4_rw(mpos, i), xp = ld4_rw(mpos, p);
      xy = static_cast<double>(x.y);
      d0 = static_cast<double>(x.x) - static_cast<double>(xp.x);
      d1 = xy - static_cast<double>(xp.y);
      d2 = static_cast<double>(x.z) - static_cast<double>(xp.z);
      unwrap_bond(L, invL, delrx, d0, d1, d2);
    }
    const bool chained = active && p == i - 1 && p >= c0;
    __syncthreads();
    if (active && p >= c0 && !chained) s_walk = 1;
    __syncthreads();
    if (s_walk) {
      // a partner inside the chunk that is not the previous bead: one by one
      s_p[tid] = p;
      s_d[0][tid] = d0;
      s_d[1][tid] = d1;
      s_d[2][tid] = d2;
      __syncthreads();
      if (tid == 0)
        for (int k = 0; k < UNWRAP_NT && c0 + k < mb.y; ++k) {
          const R4<R> up = ld4_rw(upos, s_p[k]);
          R4<R> u = ld4_rw(upos, c0 + k);
          u.x = static_cast<R>(static_cast<double>(up.x) + s_d[0][k]);
          u.y = static_cast<R>(static_cast<double>(up.y) + s_d[1][k]);
          u.z = static_cast<R>(static_cast<double>(up.z) + s_d[2][k]);
          st4(upos, c0 + k, u);
        }
      __syncthreads();
      if (active) uy = static_cast<double>(ld4_rw(upos, i).y);
    } else {
      // segment heads take their placed partner's image; a segmented scan
      // over the block adds the bond vectors down each segment
      double a0 = d0, a1 = d1, a2 = d2;
      if (active && !chained) {
        const R4<R> up = ld4_rw(upos, p);
        a0 += static_cast<double>(up.x);
        a1 += static_cast<double>(up.y);
        a2 += static_cast<double>(up.z);
      }
      int head = chained ? -1 : lane;  // inactive lanes head themselves
      for (int o = 1; o < 32; o <<= 1) {
        const int h = __shfl_up_sync(FULL, head, o);
        if (lane >= o && h > head) head = h;
      }
      for (int o = 1; o < 32; o <<= 1) {
        const double t0 = __shfl_up_sync(FULL, a0, o), t1 = __shfl_up_sync(FULL, a1, o),
                     t2 = __shfl_up_sync(FULL, a2, o);
        if (lane >= o && lane - o >= head) {  // head < 0: the segment began before the warp
          a0 += t0;
          a1 += t1;
          a2 += t2;
        }
      }
      if (lane == 31) {
        s_wsum[0][w] = a0;
        s_wsum[1][w] = a1;
        s_wsum[2][w] = a2;
        s_whead[w] = head >= 0;
      }
      __syncthreads();
      if (tid == 0) {  // carry into each warp's leading lanes, warps in order
        double c[3] = {0.0, 0.0, 0.0};
        for (int q = 0; q < NW; ++q) {
          for (int k = 0; k < 3; ++k) s_carry[k][q] = c[k];
          for (int k = 0; k < 3; ++k) c[k] = s_whead[q] ? s_wsum[k][q] : c[k] + s_wsum[k][q];
        }
      }
      __syncthreads();
      if (head < 0) {  // this lane's segment began in an earlier warp
        a0 += s_carry[0][w];
        a1 += s_carry[1][w];
        a2 += s_carry[2][w];
      }
      if (active) {
        R4<R> u = ld4_rw(upos, i);
        u.x = static_cast<R>(a0);
        u.y = static_cast<R>(a1);
        u.z = static_cast<R>(a2);
        st4(upos, i, u);
        uy = static_cast<double>(u.y);
      }
    }
    if (active) {  // the image's shear velocity
      const double ny = round((uy - xy) * invL[1]);
      R4<R> v = ld4_rw(uvel, i);
      v.x = static_cast<R>(static_cast<double>(v.x) + ny * sLy);
      st4(uvel, i, v);
    }
    __syncthreads();  // this chunk's images are placed before the next chunk reads them
  }
}

constexpr int PROF_NT = 128;   // threads per block of the profile kernels

template <typename R>
__global__ void __launch_bounds__(PROF_NT) k_profile_centre(const int2* rep_mols, const int2* mols,
                                                            const R* mpos, const R* mvel, int rep,
                                                            double* c6) {
  const int2 rm = rep_mols[rep];
  if (rm.y == 0) {
    if (threadIdx.x < 6) c6[threadIdx.x] = 0.0;
    return;
  }
  const int2 mb = mols[rm.x];
  if constexpr (std::is_same<R, double>::value) {
    __shared__ R s_stage[6][CENTRE_CHUNK];
    molecule_centre<R, PROF_NT>(mpos, mvel, mb.x, mb.y, s_stage, c6);
  } else {
    __shared__ double s_red[6 * PROF_NT], s_tot[6];
    molecule_centre_f32<PROF_NT>(mpos, mvel, mb.x, mb.y, s_red, s_tot, c6);
  }
}

// floor(x / width), x / width rounded to a double as the reference's division
// is: from x times the reciprocal, unless that is within 1e-9 of an integer
// (or past 2^20, where its error could reach that), where the division decides.
static __device__ __noinline__ long long profile_bin_div(double x, double width) {
  return static_cast<long long>(floor(x / width));
}
__device__ __forceinline__ long long profile_bin(double x, double width, double inv) {
  const double q = __dmul_rn(x, inv);
  const double magic = 6755399441055744.0;           // 1.5 2^52: floor(q) in the low bits
  const double t = __dadd_rd(q, magic);
  const double r = __dsub_rn(q, __dsub_rn(t, magic));  // in [0, 1)
  const long long k = __double2loint(t);
  if (!(r > 1e-9 && r < 1.0 - 1e-9 && k > -(1 << 20) && k < (1 << 20)))
    return profile_bin_div(x, width);
  return k;
}

// One bin's running sums in a thread's registers.
struct ProfAcc {
  long long key;
  double s0, s1;
  int n;
};
__device__ __forceinline__ void prof_flush(ProfAcc& a, double* bins) {
  if (a.n > 0) {
    atomicAdd(bins + 3 * a.key, a.s0);
    atomicAdd(bins + 3 * a.key + 1, a.s1);
    atomicAdd(bins + 3 * a.key + 2, static_cast<double>(a.n));
  }
  a.s0 = a.s1 = 0.0;
  a.n = 0;
}
__device__ __forceinline__ void prof_add(ProfAcc& even, ProfAcc& odd, long long k, long long n_bins,
                                         double v0, double v1, double* bins) {
  if (k < 0 || k >= n_bins) return;
  ProfAcc& a = (k & 1) ? odd : even;
  if (a.key != k) {
    prof_flush(a, bins);
    a.key = k;
  }
  a.s0 += v0;
  a.s1 += v1;
  ++a.n;
}

// bins: x then y, 3 doubles per bin (sum v_x, sum v_y, count), n_copies copies
// zeroed by the host; block b adds into copy b mod n_copies. Every thread
// walks `run` consecutive slots (profile_plan). The solvent is in cell order after a
// collision, so a run meets a few bins only, two neighbouring ones per axis at
// a time; their sums stay in registers (one pair for even bins, one for odd)
// and go out when the bin changes. One atomic per particle and sum onto the
// few hundred addresses took 1015 us for 1.25 M particles; this takes 115 with
// the slots in id order, where every particle changes the bin. Wraps and bins
// are decided without divisions.
template <typename R>
__global__ void __launch_bounds__(PROF_NT)
    k_velocity_profile(const RepInfo* reps, int rep, const R* rec, double delrx, double width,
                       long long kx0, int nx, long long ky0, int ny, const double* c6,
                       double* bins, int n_copies, int run) {
  const RepInfo& ri = reps[rep];
  const int i0 = (blockIdx.x * PROF_NT + threadIdx.x) * run;
  const int i1 = min(i0 + run, ri.slot_cap);
  double* bx = bins + static_cast<size_t>(blockIdx.x % n_copies) * 3 * static_cast<size_t>(nx + ny);
  double* by = bx + 3 * static_cast<size_t>(nx);
  const double c0 = c6[0], c1 = c6[1], cv0 = c6[3], cv1 = c6[4];
  const double Lx = ri.L[0], Ly = ri.L[1], inv = 1.0 / width;
  const double jump = __dmul_rn(ri.shear, Ly);
  const bool sheared = ri.shear != 0.0;
  long long lo[2], half[2], far[2];
#pragma unroll
  for (int d = 0; d < 2; ++d) {  // as make_geo: L/2 (1 - 2^-50), L/2, 1.5 L (1 - 2^-50)
    const double h = static_cast<double>(ri.L[d]) * 0.5;
    lo[d] = __double_as_longlong(h * (1.0 - 0x1.0p-50));
    half[d] = __double_as_longlong(h);
    far[d] = __double_as_longlong(3.0 * h * (1.0 - 0x1.0p-50));
  }
  ProfAcc xe{0, 0.0, 0.0, 0}, xo{1, 0.0, 0.0, 0}, ye{0, 0.0, 0.0, 0}, yo{1, 0.0, 0.0, 0};
  for (int i = i0; i < i1; ++i) {
    const size_t s = static_cast<size_t>(ri.slot_base) + i;
    const R4<R> p = ld_pos(rec, s), v = ld_vel(rec, s);
    if (slot_id(p.w) == SLOT_EMPTY) continue;
    double x0 = to_d(p.x) - c0, x1 = to_d(p.y) - c1;
    double v0 = to_d(v.x) - cv0;
    const double v1 = to_d(v.y) - cv1;
    const long long a0 = __double_as_longlong(x0) & 0x7FFFFFFFFFFFFFFFll;
    const long long a1 = __double_as_longlong(x1) & 0x7FFFFFFFFFFFFFFFll;
    if (a0 >= lo[0] || a1 >= lo[1]) {  // MPC::LEBC(pos, vel) (MPC.cpp:431-439), MPC::wrap(pos)
      if (sheared) {
        const double cy = image_d(x1, Ly, lo[1], half[1], far[1]);
        x0 = wrap_d(x0, Lx, lo[0], half[0], far[0]);
        if (cy != 0.0) {
          x0 = __dsub_rn(x0, __dmul_rn(cy, delrx));
          x1 = __dsub_rn(x1, __dmul_rn(Ly, cy));
          v0 = __dsub_rn(v0, __dmul_rn(cy, jump));
        }
        x0 = wrap_d(x0, Lx, lo[0], half[0], far[0]);
      } else {
        x0 = wrap_d(x0, Lx, lo[0], half[0], far[0]);
        x1 = wrap_d(x1, Ly, lo[1], half[1], far[1]);
      }
    }
    prof_add(xe, xo, profile_bin(x0, width, inv) - kx0, nx, v0, v1, bx);
    prof_add(ye, yo, profile_bin(x1, width, inv) - ky0, ny, v0, v1, by);
  }
  prof_flush(xe, bx);
  prof_flush(xo, bx);
  prof_flush(ye, by);
  prof_flush(yo, by);
}

// The copies of the bins into out: a warp per bin, whose lanes add every 32nd
// copy (one thread per bin added 128 of them one after the other, 19 us).
template <typename R>  // R: the precision of the instantiating unit (one copy per unit)
__global__ void k_profile_reduce(const double* bins, int n, int n_copies, double* out) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= n) return;
  double t = 0.0;
  for (int c = lane; c < n_copies; c += 32) t += bins[static_cast<size_t>(c) * n + i];
  for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xFFFFFFFFu, t, o);
  if (lane == 0) out[i] = t;
}

}  // namespace smpc

// FP32 fast-path collision kernels (the FP64 reference-parity path keeps the
// operation-by-operation kernels of mpc_kernels.cuh).
//
// Same physics as MPC::step (star-polymers/lib/Hydrodynamics/MPC.cpp:116-142),
// arranged for throughput on GB300:
//  * all per-replica constants come from a float frame written once per
//    collision (no double->float conversion in any thread: those issue on the
//    FP64 pipe, 2 lanes/clock/SM on this part);
//  * the reference's three Lees-Edwards wraps (after streaming, after the
//    grid shift, after the unshift, MPC.cpp:192-197, 301-311) are composed
//    exactly: with X = x + v h (unwrapped) the collision frame is the image
//    c_s = img(X_y + s_y) of the shifted point, the final position is the
//    image c_t = img(X_y) of the unshifted one, and the velocity picks up the
//    same total jump -(c_t) shear Ly, -(c_s) of it before the collision;
//  * k_collide takes every particle's cell from the counting sort itself
//    (sorted position -> cell range), so it never recomputes cell indices;
//  * float<->int work uses exact FP32-pipe constructions (precision.cuh).
#pragma once
#include <stdint.h>

#include "mpc_kernels.cuh"

namespace smpc {

// image index of y (-1, 0, +1) for |y| < 1.5 L; general rounding beyond
__device__ __forceinline__ float img_f(float y, float L, float half) {
  if (fabsf(y) < 1.5f * L) return y >= half ? 1.0f : (y < -half ? -1.0f : 0.0f);
  return rintf(__fdiv_rn(y, L));
}

// periodic wrap into [-L/2, L/2) for |x| < 2.5 L; general rounding beyond
__device__ __forceinline__ float wrap_f(float x, float L, float half) {
  if (!(fabsf(x) < 2.5f * L)) x = __fsub_rn(x, __fmul_rn(L, rintf(__fdiv_rn(x, L))));
  x = x >= half ? __fsub_rn(x, L) : (x < -half ? __fadd_rn(x, L) : x);
  return x >= half ? __fsub_rn(x, L) : (x < -half ? __fadd_rn(x, L) : x);
}

// The same two functions without their general-rounding branches, as
// selects: img_sel is img_f for |y| < 1.5 L, wrap_sel is wrap_f for
// |x| < 2.5 L, bit for bit (x - c L with c in {-1, 0, 1} is exact or one
// correctly rounded add either way).
__device__ __forceinline__ float img_sel(float y, float half) {
  return y >= half ? 1.0f : (y < -half ? -1.0f : 0.0f);
}
__device__ __forceinline__ float wrap_sel(float x, float L, float half) {
  x = fmaf(-img_sel(x, half), L, x);
  return fmaf(-img_sel(x, half), L, x);
}

// Recentre (MPC::check_bounds, MPC.cpp:183-188, incl. its LE wrap) and
// stream (MPC.cpp:194): X = x + v h, unwrapped. Explicitly rounded so the
// bin and collide kernels produce identical X.
__device__ __forceinline__ void stream_f(const FrameF& f, float4& x, float4& v) {
  if (f.recentre) {
    x.x = __fsub_rn(x.x, f.com[0]);
    x.y = __fsub_rn(x.y, f.com[1]);
    x.z = __fsub_rn(x.z, f.com[2]);
    v.x = __fsub_rn(v.x, f.comv[0]);
    v.y = __fsub_rn(v.y, f.comv[1]);
    v.z = __fsub_rn(v.z, f.comv[2]);
    if (f.shear_on) {
      const float c0 = img_f(x.y, f.L[1], f.half[1]);
      x.y = __fsub_rn(x.y, __fmul_rn(c0, f.L[1]));
      x.x = __fsub_rn(x.x, __fmul_rn(c0, f.delrx));
      v.x = __fsub_rn(v.x, __fmul_rn(c0, f.shearLy));
    }
  }
  x.x = __fadd_rn(x.x, __fmul_rn(v.x, f.h));
  x.y = __fadd_rn(x.y, __fmul_rn(v.y, f.h));
  x.z = __fadd_rn(x.z, __fmul_rn(v.z, f.h));
}

// Shifted collision-frame position and its y image index.
__device__ __forceinline__ float shifted_f(const FrameF& f, const float4& X, float& xs, float& ys,
                                           float& zs) {
  ys = __fadd_rn(X.y, f.shift[1]);
  const float cs = f.shear_on ? img_f(ys, f.L[1], f.half[1]) : 0.0f;
  if (f.shear_on) {
    ys = __fsub_rn(ys, __fmul_rn(cs, f.L[1]));
    xs = wrap_f(__fsub_rn(__fadd_rn(X.x, f.shift[0]), __fmul_rn(cs, f.delrx)), f.L[0], f.half[0]);
  } else {
    ys = wrap_f(ys, f.L[1], f.half[1]);
    xs = wrap_f(__fadd_rn(X.x, f.shift[0]), f.L[0], f.half[0]);
  }
  zs = wrap_f(__fadd_rn(X.z, f.shift[2]), f.L[2], f.half[2]);
  return cs;
}

__device__ __forceinline__ uint32_t cell_f(const FrameF& f, float x, float y, float z) {
  const int ix = min(f2i_floor_nonneg(fmaxf(__fadd_rn(x, f.half[0]), 0.0f)), f.Li[0] - 1);
  const int iy = min(f2i_floor_nonneg(fmaxf(__fadd_rn(y, f.half[1]), 0.0f)), f.Li[1] - 1);
  const int iz = min(f2i_floor_nonneg(fmaxf(__fadd_rn(z, f.half[2]), 0.0f)), f.Li[2] - 1);
  return static_cast<uint32_t>(ix + f.Li[0] * (iy + f.Li[1] * iz));
}

__device__ __forceinline__ float4 ld_f4(const float* p, size_t i) {
  return __ldg(reinterpret_cast<const float4*>(p) + i);
}
__device__ __forceinline__ void st_f4(float* p, size_t i, float4 v) {
  reinterpret_cast<float4*>(p)[i] = v;
}

// --------------------------------------------------------------- binning

// PACKED: 32-bit keys (local cell << 16 | rank) for contexts whose boxes
// have at most 65,536 cells each, half the bytes of the (global cell, rank)
// pairs between the binning and the permutation. A cell of 65,535 particles
// or more cannot be packed and raises ERR_KEY_MISMATCH.
template <int NT, int U, bool PACKED>
__global__ void __launch_bounds__(NT) k_fluid_bin_f32(const Tile* tiles, const RepInfo* reps,
                                                      const FrameF* frames,
                                                      const float* __restrict__ st,
                                                      uint2* __restrict__ keys, uint32_t* count,
                                                      ErrorState* err) {
  const Tile t = tiles[blockIdx.x];
  const FrameF f = frames[t.rep];
  const uint32_t cbase = static_cast<uint32_t>(reps[t.rep].cell_base);
  const unsigned lane = threadIdx.x & 31u;
  const unsigned below = (1u << lane) - 1u;
  for (int base = t.begin; base < t.end; base += NT * U) {
    float4 x[U], v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = base + u * NT + threadIdx.x;
      if (i < t.end) {
        x[u] = ld_f4(st, 2 * static_cast<size_t>(i));
        v[u] = ld_f4(st, 2 * static_cast<size_t>(i) + 1);
      }
    }
    uint32_t key[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = base + u * NT + threadIdx.x;
      key[u] = KEY_NONE;
      if (i < t.end && __float_as_uint(x[u].w) != SLOT_EMPTY) {
        stream_f(f, x[u], v[u]);
        float xs, ys, zs;
        shifted_f(f, x[u], xs, ys, zs);
        key[u] = cbase + cell_f(f, xs, ys, zs);
      }
    }
    unsigned peers[U];
    uint32_t rbase[U];
#pragma unroll
    for (int u = 0; u < U; ++u) peers[u] = __match_any_sync(0xFFFFFFFFu, key[u]);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      rbase[u] = 0u;
      if (lane == static_cast<unsigned>(__ffs(peers[u]) - 1) && key[u] != KEY_NONE)
        rbase[u] = atomicAdd(count + key[u], __popc(peers[u]));
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t b0 = __shfl_sync(0xFFFFFFFFu, rbase[u], __ffs(peers[u]) - 1);
      const int i = base + u * NT + threadIdx.x;
      if (i >= t.end) continue;
      const uint32_t rank = b0 + __popc(peers[u] & below);
      if (PACKED) {
        uint32_t k32 = KEY_NONE;
        if (key[u] != KEY_NONE) {
          if (rank >= 0xFFFFu)
            raise_error(err, ERR_KEY_MISMATCH, static_cast<uint32_t>(i), key[u]);
          else
            k32 = ((key[u] - cbase) << 16) | rank;
        }
        reinterpret_cast<uint32_t*>(keys)[i] = k32;
      } else {
        keys[i] = make_uint2(key[u], rank);
      }
    }
  }
}

// --------------------------------------------------------------- collide

// A staged particle: sx = (X unwrapped streamed position, id or MONO_BIT|m),
// sv = (velocity in the collision frame, mass).
struct FastP {
  float4 x;
  float4 v;
};

__device__ __forceinline__ void fetch_f(FastP& P, uint32_t src, const float* st,
                                        const float* mpos, const float* mvel, const int* mimg,
                                        const FrameF& f, int wrap_mono) {
  if (src & MONO_BIT) {
    const uint32_t m = src & ~MONO_BIT;
    P.v = reinterpret_cast<const float4*>(mvel)[m];
    P.v.w = reinterpret_cast<const float4*>(mpos)[m].w;
    if (wrap_mono == MONOBIN_WRAPPED)
      P.v.x = __fsub_rn(P.v.x, __fmul_rn(i2f_small(mimg[m]), f.shearLy));
    P.x = make_float4(0.f, 0.f, 0.f, __uint_as_float(src));
  } else {
    P.x = ld_f4(st, 2 * static_cast<size_t>(src));
    P.v = ld_f4(st, 2 * static_cast<size_t>(src) + 1);
  }
}

// Solvent: stream (the unwrapped X replaces the position, the id stays in
// .w) and move the velocity into the shifted collision frame (image c_s).
// Monomers keep what fetch_f loaded.
__device__ __forceinline__ void frame_f(FastP& P, const FrameF& f, float solvent_mass) {
  if (__float_as_uint(P.x.w) & MONO_BIT) return;
  stream_f(f, P.x, P.v);
  if (f.shear_on) {
    const float cs = img_f(__fadd_rn(P.x.y, f.shift[1]), f.L[1], f.half[1]);
    P.v.x = __fsub_rn(P.v.x, __fmul_rn(cs, f.shearLy));
  }
  P.v.w = solvent_mass;
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

// One solvent slot record (32 bytes) in one 256-bit store.
__device__ __forceinline__ void st_rec_f(float* st, size_t slot, float x, float y, float z,
                                         float w, float vx, float vy, float vz) {
  asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(st + 8 * slot), "f"(x),
               "f"(y), "f"(z), "f"(w), "f"(vx), "f"(vy), "f"(vz), "f"(0.0f)
               : "memory");
}

// Rarely taken code of the collide, out of line, so that the instructions
// which every tile executes stay together: with all of it inlined the kernel
// was 61 KB, and its warps waited for instruction fetches a fifth of the time.
static __device__ __noinline__ void raise_cold(ErrorState* e, uint32_t bit, uint32_t a, uint32_t b) {
  raise_error(e, bit, a, b);
}
static __device__ __noinline__ float img_far(float y, float L) { return rintf(__fdiv_rn(y, L)); }
__device__ __forceinline__ float img_c(float y, float L, float half) {
  if (fabsf(y) < 1.5f * L) return img_sel(y, half);
  return img_far(y, L);
}
static __device__ __noinline__ float wrap_far(float x, float L) {
  return __fsub_rn(x, __fmul_rn(L, img_far(x, L)));
}
__device__ __forceinline__ float wrap_c(float x, float L, float half) {
  if (!(fabsf(x) < 2.5f * L)) x = wrap_far(x, L);
  return wrap_sel(x, L, half);
}
// The draws' functions, one copy each for both kinds of draw.
static __device__ __noinline__ Uniform2<float> draw_uniforms(unsigned long long seed, uint32_t cell,
                                                             unsigned long long step, uint32_t k) {
  return philox_uniforms<float>(seed, cell, step, k);
}
static __device__ __noinline__ float2 sincos_turns(float u) {
  float2 r;
  sincosf(6.283185307179586f * u, &r.x, &r.y);
  return r;
}
static __device__ __noinline__ bool gamma_accept(float u, float x2, float d, float v) {
  return logf(u) < 0.5f * x2 + d * (1.0f - v + logf(v));
}
// philox_gamma<float> (philox.cuh) on the functions above
__device__ __forceinline__ float cell_gamma(unsigned long long seed, uint32_t cl,
                                            unsigned long long step, uint32_t nn, bool* ok) {
  const float d = 1.5f * i2f_small(static_cast<int>(nn - 1u)) - 1.0f / 3.0f;
  const float c = 1.0f / sqrtf(9.0f * d);
#pragma unroll 1
  for (uint32_t it = 0; it < 64u; ++it) {
    const Uniform2<float> n = draw_uniforms(seed, cl, step, 1u + 2u * it);
    const float x = sqrtf(-2.0f * logf(n.a)) * sincos_turns(n.b).y;
    float v = 1.0f + c * x;
    if (v <= 0.0f) continue;
    v = v * v * v;
    const float u = draw_uniforms(seed, cl, step, 2u + 2u * it).a;
    const float x2 = x * x;
    if (u < 1.0f - 0.0331f * (x2 * x2) || gamma_accept(u, x2, d, v)) return d * v;
  }
  *ok = false;
  return d;
}

// Two FP32 operations in one instruction, each rounded by itself. (A packed
// multiply whose result is added comes out contracted, whatever its rounding
// is called; only products that feed an fma's factor are packed here.)
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// fix32_add (precision.cuh) of two values
__device__ __forceinline__ void fix32_add2(f32x2 v, uint32_t& ha, uint32_t& la, uint32_t& hb,
                                           uint32_t& lb) {
  const f32x2 magic = pack2(12582912.0f, 12582912.0f), s10 = pack2(1024.0f, 1024.0f);
  const f32x2 m = fma2(v, s10, magic);
  const f32x2 r = fma2(v, s10, fma2(m, pack2(-1.0f, -1.0f), magic));
  const f32x2 l = fma2(r, pack2(4194304.0f, 4194304.0f), magic);
  float m0, m1, l0, l1;
  unpack2(m, m0, m1);
  unpack2(l, l0, l1);
  ha += __float_as_uint(m0);
  hb += __float_as_uint(m1);
  la += __float_as_uint(l0);
  lb += __float_as_uint(l1);
}

// The cell arithmetic of the collide, with every contraction written out, so
// that a cell's result does not depend on what the code is inlined into.
// Per particle: m |v|^2 / 256 (mq = m / 256).
__device__ __forceinline__ float cell_energy_term(float mq, float x, float y, float z) {
  return __fmul_rn(mq, __fmaf_rn(z, z, __fmaf_rn(x, x, __fmul_rn(y, y))));
}
// kinetic energy about the cell velocity: S is the sum of the terms above, q
// the cell's momentum, inv its inverse mass
__device__ __forceinline__ float cell_ekin(float S, float q0, float q1, float q2, float inv) {
  const float qq = __fmaf_rn(q2, q2, __fmaf_rn(q0, q0, __fmul_rn(q1, q1)));
  return fmaxf(__fmul_rn(0.5f, __fmaf_rn(S, 256.0f, -__fmul_rn(qq, inv))), 0.0f);
}
// rows of the rotation about the axis a (MPC.cpp:244-257)
__device__ __forceinline__ void cell_rows(float a0, float a1, float a2, float c, float s,
                                          float4* rows) {
  const float oc = __fsub_rn(1.0f, c);
  const float p00 = __fmul_rn(a0, a0), p11 = __fmul_rn(a1, a1), p22 = __fmul_rn(a2, a2);
  const float p01 = __fmul_rn(a0, a1), p02 = __fmul_rn(a0, a2), p12 = __fmul_rn(a1, a2);
  rows[0] = make_float4(__fmaf_rn(__fsub_rn(1.0f, p00), c, p00),
                        __fmaf_rn(p01, oc, -__fmul_rn(a2, s)), __fmaf_rn(a1, s, __fmul_rn(p02, oc)),
                        0.0f);
  rows[1] = make_float4(__fmaf_rn(p01, oc, __fmul_rn(a2, s)),
                        __fmaf_rn(__fsub_rn(1.0f, p11), c, p11),
                        __fmaf_rn(p12, oc, -__fmul_rn(a0, s)), 0.0f);
  rows[2] = make_float4(__fmaf_rn(-a1, s, __fmul_rn(p02, oc)), __fmaf_rn(p12, oc, __fmul_rn(a0, s)),
                        __fmaf_rn(__fsub_rn(1.0f, p22), c, p22), 0.0f);
}
struct CellSums {
  long long px, py, pz, e;
  int nsol;
  float mmono;
  uint32_t top;
};
__device__ __forceinline__ void recentre_c(const FrameF& f, float4& x, float4& v) {
  x.x = __fsub_rn(x.x, f.com[0]);
  x.y = __fsub_rn(x.y, f.com[1]);
  x.z = __fsub_rn(x.z, f.com[2]);
  v.x = __fsub_rn(v.x, f.comv[0]);
  v.y = __fsub_rn(v.y, f.comv[1]);
  v.z = __fsub_rn(v.z, f.comv[2]);
  if (f.shear_on) {
    const float c0 = img_c(x.y, f.L[1], f.half[1]);
    x.y = __fsub_rn(x.y, __fmul_rn(c0, f.L[1]));
    x.x = __fsub_rn(x.x, __fmul_rn(c0, f.delrx));
    v.x = __fsub_rn(v.x, __fmul_rn(c0, f.shearLy));
  }
}
static __device__ __noinline__ FastP fetch_frame_cold(uint32_t src, const float* st,
                                                      const float* mpos, const float* mvel,
                                                      const int* mimg, const FrameF& f,
                                                      int mono_bin) {
  FastP P;
  fetch_f(P, src, st, mpos, mvel, mimg, f, mono_bin);
  frame_f(P, f, f.solvent_mass);
  return P;
}
// The largest fixed-point term of every second staged particle of mass m from j
// to j1 (NaN terms are not terms: they raise ERR_NONFINITE later).
static __device__ __noinline__ uint32_t largest_term(const float4* v, int j, int j1, float m) {
  float big = 0.0f;
  for (; j < j1; j += 2) {
    const float et = cell_energy_term(m * 0.00390625f, v[j].x, v[j].y, v[j].z);
    big = fmaxf(big, fmaxf(fmaxf(fabsf(v[j].x * m), fabsf(v[j].y * m)), fmaxf(fabsf(v[j].z * m), et)));
  }
  return __float_as_uint(big);
}
// A particle's copies where monomers are among the warp's particles.
static __device__ __noinline__ void copy_mixed(uint32_t src, float4* x, float4* v, const float* st,
                                               const float* mvel) {
  if (src & MONO_BIT) {
    *x = make_float4(0.f, 0.f, 0.f, __uint_as_float(src));
    cp_async16(v, mvel + 4 * static_cast<size_t>(src & ~MONO_BIT));
  } else {
    cp_async16(x, st + 8 * static_cast<size_t>(src));
    cp_async16(v, st + 8 * static_cast<size_t>(src) + 4);
  }
}
// Every second particle of a cell from sorted position j (tile-local) to j1,
// read from global memory: a tile's particles past the staging capacity.
static __device__ __noinline__ CellSums cell_overflow(int j, int j1, uint32_t p0, const float* st,
                                                      const float* mpos, const float* mvel,
                                                      const int* mimg, const uint32_t* perm,
                                                      const FrameF& f, int mono_bin) {
  CellSums o = {0, 0, 0, 0, 0, 0.0f, 0u};
  for (; j < j1; j += 2) {
    const uint32_t src = perm[p0 + j];
    const FastP P = fetch_frame_cold(src, st, mpos, mvel, mimg, f, mono_bin);
    const float mx = P.v.x * P.v.w, my = P.v.y * P.v.w, mz = P.v.z * P.v.w;
    const float et = cell_energy_term(P.v.w * 0.00390625f, P.v.x, P.v.y, P.v.z);
    const float big = fmaxf(fmaxf(fabsf(mx), fabsf(my)), fmaxf(fabsf(mz), et));
    o.top = max(o.top, __float_as_uint(fmaxf(big, 0.0f)));
    o.px += f2fix32(mx);
    o.py += f2fix32(my);
    o.pz += f2fix32(mz);
    o.e += f2fix32(et);
    if (src & MONO_BIT) {
      o.mmono += P.v.w;
    } else {
      ++o.nsol;
    }
  }
  return o;
}
__device__ __forceinline__ float row_apply(const float4& r, float d0, float d1, float d2) {
  return __fadd_rn(r.w, __fmaf_rn(r.z, d2, __fmaf_rn(r.x, d0, __fmul_rn(r.y, d1))));
}

// One CTA of two warps per tile of up to COL_CT cells of one replica.
//  gather : sorted slots, then the records by cp.async straight into shared
//           memory (no registers and no L1 lines held while they are on their
//           way; a gather through registers was limited by the L1 lines left
//           beside the staging buffer and ran 1.4x slower);
//  draws  : while the records arrive, one lane per cell: the first warp the
//           gamma variates, the second the rotations (neither needs the
//           particles), each in a full warp without divergence;
//  frame  : every warp streams the particles it copied and moves them into
//           the collision frame, in place;
//  cells  : two lanes per cell, int64 2^32 fixed-point sums (exact, so
//           independent of the particles' order), then the thermostat factor,
//           folded into the cell's rotation;
//  apply  : v' = cmv + sR (v - cmv), back to the primary box, written in cell
//           order as 32-byte records.
// What bounds it: instruction issue (60 % of the slots; 11.1 warp
// instructions per particle), then the latency of the phases. Small CTAs keep
// more of them in different phases and their barriers cheap: 16 CTAs of 64
// threads and 32 cells fit one SM and ran at 935 us for 65.8 M particles,
// 8 CTAs of 128 threads and 64 cells at 980 us, the kernel before (draws after
// the sums, two copies per record, everything inlined) at 1073 us; 4.5 GB of
// records, slots and offsets, so 4.8 TB/s.
constexpr int COL_NT = 64;    // threads
constexpr int COL_CT = 32;    // cells per tile at most: two lanes each
constexpr int COL_CAP = 360;  // staged particles; the rest is read from global memory again
__global__ void __launch_bounds__(COL_NT, 15) k_collide_tile(
    const Tile* tiles, const RepInfo* reps, const FrameF* __restrict__ frames, const RepDyn* dyn,
    const uint32_t* __restrict__ off, const uint32_t* __restrict__ perm,
    const float* __restrict__ st_in, float* __restrict__ st_out, const float* mpos, float* mvel,
    const int* mimg, const double* inj_gamma, const double* inj_uphi, const double* inj_utheta,
    int rng, int mono_bin, ErrorState* err) {
  constexpr unsigned FULL = 0xFFFFFFFFu;
  constexpr int NT = COL_NT, CT = COL_CT, CAP = COL_CAP;
  static_assert(NT == 2 * CT && NT == 64, "two lanes per cell; one warp per kind of draw");
  constexpr int J = (CAP + NT - 1) / NT;  // staged particles per thread
  __shared__ float4 s_x[CAP];      // streamed position, id (or MONO_BIT | monomer)
  __shared__ float4 s_v[CAP];      // velocity in the collision frame, then the cell in .w
  __shared__ float4 s_rc[CT * 3];  // per cell: rows of sR, cell velocity in .w
  __shared__ float s_g[CT];        // per cell: gamma variate
  __shared__ uint32_t s_off[CT + 1];

  const Tile t = tiles[blockIdx.x];
  const int nc = t.end - t.begin;
  for (int i = threadIdx.x; i <= nc; i += NT) s_off[i] = off[t.begin + i];
  __syncthreads();
  const uint32_t p0 = s_off[0];
  const int n = static_cast<int>(s_off[nc] - p0);
  const int nloc = n < CAP ? n : CAP;

  int mono = 0;
  {
    uint32_t src[J];
#pragma unroll
    for (int u = 0; u < J; ++u) {
      const int j = u * NT + threadIdx.x;
      src[u] = j < nloc ? perm[p0 + j] : 0xFFFFFFFFu;
    }
    // Two lanes per record, one for each 16-byte half, so that a copy
    // instruction touches every record's 128-byte line and 32-byte sector once
    const int part = static_cast<int>(threadIdx.x & 1u);
    const int l0 = static_cast<int>((threadIdx.x & 31u) >> 1);
    const int w0 = static_cast<int>(threadIdx.x & ~31u);
    float4* dst = (part ? s_v : s_x) + w0 + l0;
    const float* from = st_in + 4 * part;
#pragma unroll
    for (int u = 0; u < J; ++u) {
      if (u * NT + w0 >= nloc) break;  // whole warps
      const int j = u * NT + static_cast<int>(threadIdx.x);
      if (!__any_sync(FULL, (src[u] & MONO_BIT) && j < nloc)) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const uint32_t sr = __shfl_sync(FULL, src[u], 16 * k + l0);
          if (u * NT + 16 * k + w0 + l0 < nloc)
            cp_async16(dst + u * NT + 16 * k, from + 8 * static_cast<size_t>(sr));
        }
      } else {
        mono = 1;
        if (j < nloc) copy_mixed(src[u], s_x + j, s_v + j, st_in, mvel);
      }
    }
  }
  const FrameF& f = frames[t.rep];
  // the cells' draws while the records are on their way
  {
    const RepInfo& ri = reps[t.rep];
    const uint32_t cbase = static_cast<uint32_t>(ri.cell_base);
    const unsigned long long seed = ri.seed;
    const unsigned long long step = dyn[t.rep].step;
    const bool axis = threadIdx.x >= 32;
    const int c = static_cast<int>(threadIdx.x & 31u);
    if (c < nc) {
      const uint32_t cg = static_cast<uint32_t>(t.begin + c), cl = cg - cbase;
      if (axis) {
        float uphi, a2;
        if (rng == RNG_INJECT) {
          uphi = static_cast<float>(inj_uphi[cg]);
          a2 = 2.0f * (static_cast<float>(inj_utheta[cg]) - 0.5f);
        } else {
          const Uniform2<float> u = draw_uniforms(seed, cl, step, 0u);
          uphi = u.a;
          a2 = 2.0f * (u.b - 0.5f);
        }
        const float r = sqrtf(__fmaf_rn(-a2, a2, 1.0f));
        const float2 sc = sincos_turns(uphi);
        cell_rows(r * sc.y, r * sc.x, a2, f.rot_c, f.rot_s, s_rc + 3 * c);
      } else {
        const uint32_t nn = s_off[c + 1] - s_off[c];
        float gv = 1.0f;
        if (nn >= 2u) {
          if (rng == RNG_INJECT) {
            gv = static_cast<float>(inj_gamma[cg]);
          } else {
            bool ok = true;
            gv = cell_gamma(seed, cl, step, nn, &ok);
            if (!ok) raise_cold(err, ERR_GAMMA_ITERS, cg, nn);
            gv *= f.kT;
          }
        }
        s_g[c] = gv;
      }
    }
  }
  {
    const bool recentre = f.recentre != 0, shear_on = f.shear_on != 0;
    const float h = f.h, sh1 = f.shift[1], L1 = f.L[1], half1 = f.half[1], sLy = f.shearLy;
    cp_async_wait_all();
    __syncwarp();  // a warp finishes the particles that its lanes copied
    // stream and move into the collision frame, in place
#pragma unroll 1
    for (int j = threadIdx.x; j < nloc; j += NT) {
      float4 x = s_x[j], v = s_v[j];
      if (__float_as_uint(x.w) & MONO_BIT) {
        const uint32_t m = __float_as_uint(x.w) & ~MONO_BIT;
        v.w = reinterpret_cast<const float4*>(mpos)[m].w;
        if (mono_bin == MONOBIN_WRAPPED)
          v.x = __fsub_rn(v.x, __fmul_rn(i2f_small(mimg[m]), sLy));
        s_v[j] = v;
        continue;
      }
      if (recentre) {
        recentre_c(f, x, v);
        s_v[j] = v;
      }
      x.x = __fadd_rn(x.x, __fmul_rn(v.x, h));
      x.y = __fadd_rn(x.y, __fmul_rn(v.y, h));
      x.z = __fadd_rn(x.z, __fmul_rn(v.z, h));
      s_x[j] = x;
      const float ys = __fadd_rn(x.y, sh1);
      if (shear_on && !(fabsf(ys) < half1))  // at or past a y face (or NaN)
        s_v[j].x = __fsub_rn(v.x, __fmul_rn(img_c(ys, L1, half1), sLy));
    }
  }
  mono = __syncthreads_or(mono);

  // cells: two lanes each; int64 2^32 fixed-point sums (exact, order-free)
  {
    const int lc = threadIdx.x >> 1;
    const int half = threadIdx.x & 1;
    const bool live = lc < nc;
    const int j0 = live ? static_cast<int>(s_off[lc] - p0) : 0;
    const int j1 = live ? static_cast<int>(s_off[lc + 1] - p0) : 0;
    const float ms = f.solvent_mass;
    long long px = 0, py = 0, pz = 0, e = 0;
    int nsol = 0;
    float mmono = 0.0f;
    const int jl = j1 < nloc ? j1 : nloc;  // staged part of the cell
    const float tag = __int_as_float(lc);
    // Largest fixed-point term, as bits. Without monomers and for masses below
    // 15, m |v|^2 / 256 is the largest term of any particle past the limit.
    uint32_t top = 0;
    const bool pure = !mono && ms < 15.0f;
    {
      uint32_t xh = 0, xl = 0, yh = 0, yl = 0, zh = 0, zl = 0, eh = 0, el = 0;
      int terms = 0;
      if (pure) {
        const float mq = ms * 0.00390625f;
        // the next particle is loaded before this one's tag is stored (the
        // store may alias the load as far as the compiler knows)
        float4 v = s_v[j0 + half < jl ? j0 + half : 0];
#pragma unroll 1
        for (int j = j0 + half; j < jl; j += 2) {
          const float4 next = s_v[j + 2 < jl ? j + 2 : j];
          s_v[j].w = tag;
          const float et = cell_energy_term(mq, v.x, v.y, v.z);
          top = max(top, __float_as_uint(et));
          fix32_add2(mul2(pack2(v.x, v.y), pack2(ms, ms)), xh, xl, yh, yl);
          fix32_add2(pack2(v.z * ms, et), zh, zl, eh, el);
          ++terms;
          v = next;
        }
        nsol = terms;
      } else {
#pragma unroll 1
        for (int j = j0 + half; j < jl; j += 2) {
          const float4 v = s_v[j];
          const bool is_mono = __float_as_uint(s_x[j].w) & MONO_BIT;
          s_v[j].w = tag;
          const float m = is_mono ? v.w : ms;
          const float mx = v.x * m, my = v.y * m, mz = v.z * m;
          const float et = cell_energy_term(m * 0.00390625f, v.x, v.y, v.z);
          const float big = fmaxf(fmaxf(fabsf(mx), fabsf(my)), fmaxf(fabsf(mz), et));
          top = max(top, __float_as_uint(fmaxf(big, 0.0f)));
          fix32_add(mx, xh, xl);
          fix32_add(my, yh, yl);
          fix32_add(mz, zh, zl);
          fix32_add(et, eh, el);
          ++terms;
          if (is_mono) {
            mmono += m;
          } else {
            ++nsol;
          }
        }
      }
      px = fix32_join(xh, xl, terms);
      py = fix32_join(yh, yl, terms);
      pz = fix32_join(zh, zl, terms);
      e = fix32_join(eh, el, terms);
    }
    uint32_t over = 0;  // largest term past the staging capacity
    if (n > nloc) {
      const CellSums o = cell_overflow((j0 > nloc ? j0 : nloc) + half, j1, p0, st_in, mpos, mvel, mimg,
                                       perm, f, mono_bin);
      px += o.px;
      py += o.py;
      pz += o.pz;
      e += o.e;
      nsol += o.nsol;
      mmono += o.mmono;
      over = o.top;
    }
    const uint32_t cg = static_cast<uint32_t>(t.begin + lc);
    if (max(top, over) >= __float_as_uint(FIX32_LIMIT)) {
      if (pure) top = largest_term(s_v, j0 + half, jl, ms);  // without the NaN among them
      top = max(top, over);
      if (top >= __float_as_uint(FIX32_LIMIT)) raise_cold(err, ERR_FIXPOINT, cg, top);
    }
    px += __shfl_xor_sync(FULL, px, 1);
    py += __shfl_xor_sync(FULL, py, 1);
    pz += __shfl_xor_sync(FULL, pz, 1);
    e += __shfl_xor_sync(FULL, e, 1);
    nsol += __shfl_xor_sync(FULL, nsol, 1);
    if (mono || n > nloc) mmono += __shfl_xor_sync(FULL, mmono, 1);
    if (live) {
      const uint32_t nn = static_cast<uint32_t>(j1 - j0);
      const float mt = fmaf(i2f_small(nsol), ms, mmono);
      const float inv = mt > 0.f ? 1.0f / mt : 0.0f;
      const float q0 = fix32_to_f(px), q1 = fix32_to_f(py), q2 = fix32_to_f(pz);
      const float ekin = cell_ekin(fix32_to_f(e), q0, q1, q2, inv);
      // (an injected variate without a square root: no thermostat)
      const float factor = nn >= 2u && ekin > 0.f ? sqrtf(s_g[lc] / ekin) : 1.0f;
      const float sc = factor >= 0.0f ? factor : 1.0f;
#pragma unroll
      for (int r = 0; r < 3; r += 2) {  // rows 0 and 2 on the even lane, 1 on the odd one
        const int row = r + half;
        if (row > 2) break;
        float4 m = s_rc[3 * lc + row];
        m.x = __fmul_rn(m.x, sc);
        m.y = __fmul_rn(m.y, sc);
        m.z = __fmul_rn(m.z, sc);
        m.w = (row == 0 ? q0 : row == 1 ? q1 : q2) * inv;
        s_rc[3 * lc + row] = m;
      }
    }
  }
  __syncthreads();

  // apply: v' = cmv + sR (v - cmv), back to the primary box, write in cell order
  const float hx = f.half[0], hy = f.half[1], hz = f.half[2], sh1 = f.shift[1];
#pragma unroll 1
  for (int j = threadIdx.x; j < n; j += NT) {
    float4 x, v;
    int c;
    if (j < nloc) {
      x = s_x[j];
      v = s_v[j];
      c = __float_as_int(v.w);
    } else {  // past the staging capacity
      const FastP P = fetch_frame_cold(perm[p0 + j], st_in, mpos, mvel, mimg, f, mono_bin);
      x = P.x;
      v = P.v;
      c = 0;  // the cell whose range holds sorted position p0 + j
      while (static_cast<int>(s_off[c + 1] - p0) <= j) ++c;
    }
    const float4 r0 = s_rc[3 * c], r1 = s_rc[3 * c + 1], r2 = s_rc[3 * c + 2];
    const float d0 = v.x - r0.w, d1 = v.y - r1.w, d2 = v.z - r2.w;
    float vx = row_apply(r0, d0, d1, d2);
    const float vy = row_apply(r1, d0, d1, d2);
    const float vz = row_apply(r2, d0, d1, d2);
    const uint32_t tag = __float_as_uint(x.w);
    if (!(isfinite(vx) && isfinite(vy) && isfinite(vz))) raise_cold(err, ERR_NONFINITE, p0 + j, tag);
    const size_t p = static_cast<size_t>(p0) + j;
    if (tag & MONO_BIT) {
      const uint32_t m = tag & ~MONO_BIT;
      if (mono_bin == MONOBIN_WRAPPED) vx = __fadd_rn(vx, __fmul_rn(i2f_small(mimg[m]), f.shearLy));
      float4 mv = reinterpret_cast<float4*>(mvel)[m];
      mv.x = vx;
      mv.y = vy;
      mv.z = vz;
      reinterpret_cast<float4*>(mvel)[m] = mv;
      st_rec_f(st_out, p, 0.f, 0.f, 0.f, __uint_as_float(SLOT_EMPTY), 0.f, 0.f, 0.f);
      continue;
    }
    float X = x.x, Y = x.y, Z = x.z;
    const float ys = __fadd_rn(Y, sh1);
    if (!(fabsf(X) < hx && fabsf(Y) < hy && fabsf(ys) < hy && fabsf(Z) < hz)) {
      // final image c_t of the streamed point; the velocity already carries -c_s
      const float cs = f.shear_on ? img_c(ys, f.L[1], f.half[1]) : 0.0f;
      if (f.shear_on) {
        const float ct = img_c(Y, f.L[1], f.half[1]);
        Y = __fsub_rn(Y, __fmul_rn(ct, f.L[1]));
        X = wrap_c(__fsub_rn(X, __fmul_rn(ct, f.delrx)), f.L[0], f.half[0]);
        vx = __fsub_rn(vx, __fmul_rn(ct - cs, f.shearLy));
      } else {
        X = wrap_c(X, f.L[0], f.half[0]);
        Y = wrap_c(Y, f.L[1], f.half[1]);
      }
      Z = wrap_c(Z, f.L[2], f.half[2]);
    }
    st_rec_f(st_out, p, X, Y, Z, x.w, vx, vy, vz);
  }
}

}  // namespace smpc

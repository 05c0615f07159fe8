// Tile kernel of the solid with one element row per thread (tiles by rows of
// sf2d_tiler.h): thread 5 e + j of a CTA advances row j of element e, five
// points with both components.
//
// The mapping, the moduli and the row of every derivative, stress and
// transpose stay in the thread's registers; only the displacement of the
// element and the gamma half of the weak-form terms pass through shared memory
// once.  Tasks of rows, columns and points that hand every intermediate over
// through shared memory are bound by that traffic and by their barriers; a
// whole element in one or two threads' registers needs fewer operations, but
// leaves too few warps in flight and is slower on every mesh but the largest.
//
// What bounds it: latency at 19 warps per SM (1000 x 400 elements: issue slots
// half used, DRAM at 3.6 of 6.55 TB/s); with attenuation on large meshes DRAM
// (1600 x 800 elements: 5.0 GB in 0.855 ms, 5.9 TB/s).  So all that does not
// change from step to step is requested before the previous kernel is waited
// for: the element data, the largest part of the bytes, into registers, the
// inverse mass and the lists of shared points by cp.async, and what is read and
// written in place into L2.
//
// Per step, against tasks of rows, columns and points (tiles of 32 elements):
// 80 x 60 elements 10.9 -> 9.9 us, 233 x 147 with topography 21.4 -> 17.9 us,
// 1000 x 400 187 -> 172 us, 301 x 199 anisotropic 46.4 -> 32.4 us, 800 x 400
// attenuating 323 -> 242 us, 301 x 150 attenuating with LDDRK 490 -> 403 us.
//
// Derivatives are taken of the differences to the element's centre
// value, where the field's large common part cancels before anything is
// rounded; the row sums of the derivative matrix, zero but for its
// coefficients' rounding, times the centre value keep the given matrix.  No
// factor is folded into another on the host (the Jacobian or the weights into
// the moduli): a rounded product is the same in every step, and its effect
// grows with the steps where rounding that varies averages out.
//
// Phases of one CTA (a tile):
//   1. cp.async of the fields of the tile's points into shared memory;
//   2. Newmark predictor; the interior points' displacement is final here and
//      is written at once;
//   3. Stacey, coupling and source terms (one thread per receiving point);
//   4. the element rows: differences to the centre into the element's array;
//      derivatives along the row and, from the array, across it; stress (with
//      anisotropy or 3-SLS memory variables), kernel integrands of an adjoint
//      run, weak-form terms; the gamma terms through a second array; weighted
//      transposes;
//   5. assembly into the shared accumulator, phase by phase (TileInfo::ncol,
//      four in meshes of one orientation), without atomics;
//   6. mass, corrector or LDDRK update, write-back; the shared points' partial
//      sums for the kernel that finishes them.
// Results are bit-identical from run to run.
#pragma once

#include "sf2d_kernels.cuh"

namespace sf2d {

// Shared memory of a tile by rows: u, v, acc, inverse mass or partial-sum slot
// (and the forward frame) of its points; per element 25 differences to the
// centre (and the frame's) and 25 gamma terms (stride 25 float2: the elements
// of a warp fall into different banks; rows padded for 16-byte accesses take
// 183 instead of 170 us at 1000 x 400 elements); the line matrices.
struct RowSmem {
  size_t v, acc, rm, b, w, wb, t, h, total;
};
__host__ __device__ inline RowSmem row_smem_layout(int max_local, int max_elems, bool kern) {
  const size_t lb = align16(static_cast<size_t>(max_local) * sizeof(float2));
  const size_t eb = align16(static_cast<size_t>(max_elems) * 25 * sizeof(float2));
  RowSmem L;
  L.v = lb;
  L.acc = 2 * lb;
  L.rm = 3 * lb;
  L.b = 4 * lb;
  L.w = L.b + (kern ? lb : 0);
  L.wb = L.w + eb;
  L.t = L.wb + (kern ? eb : 0);
  L.h = L.t + eb;
  L.total = L.h + 64 * sizeof(float);
  return L;
}

// Requests a range of global memory into L2 (the whole 16-byte units in it).
__device__ __forceinline__ void prefetch_l2(const void *p, size_t bytes) {
  const size_t a = (reinterpret_cast<size_t>(p) + 15) & ~static_cast<size_t>(15), b = (reinterpret_cast<size_t>(p) + bytes) & ~static_cast<size_t>(15);
  if (a < b) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(a), "r"(static_cast<unsigned>(b - a)) : "memory");
}

// a * h + c, both components in one instruction
__device__ __forceinline__ float2 f2_fma2(float2 a, float2 hh, float2 c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(d)
      : "l"(*reinterpret_cast<unsigned long long *>(&a)), "l"(*reinterpret_cast<unsigned long long *>(&hh)),
        "l"(*reinterpret_cast<unsigned long long *>(&c)));
  return *reinterpret_cast<float2 *>(&d);
}
__device__ __forceinline__ float2 f2_sub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 f2_fma(float2 a, float h, float2 c) { return make_float2(fmaf(a.x, h, c.x), fmaf(a.y, h, c.y)); }

// Derivatives along a row, out[m] = sum_k h[m][k] u[k], from the differences w
// to the centre value uc, and the weighted transposes out[m] = sum_k
// hprimewgll[k][m] t[k].  The given coefficients are used as they are: even
// and odd parts would save a fifth of the operations, but the rounding of
// their combined coefficients is the same in every element and step and
// shifts the wave speed by more than the rounding of the fields does.
__device__ __forceinline__ void row_derivs(const Params &P, const float2 (&w)[5], float2 uc, float2 (&out)[5]) {
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    float2 d = make_float2(uc.x * P.hsum[m], uc.y * P.hsum[m]);
#pragma unroll
    for (int k = 0; k < 5; ++k) d = f2_fma(w[k], P.hconst[5 * m + k], d);
    out[m] = d;
  }
}
__device__ __forceinline__ void row_transposed(const Params &P, const float2 (&t)[5], float2 (&out)[5]) {
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    float2 d = make_float2(t[0].x * P.hconst[25 + m], t[0].y * P.hconst[25 + m]);
#pragma unroll
    for (int k = 1; k < 5; ++k) d = f2_fma(t[k], P.hconst[25 + 5 * k + m], d);
    out[m] = d;
  }
}

// Memory-variable update of one element point (Newmark recursive convolution or
// LDDRK ADE stage, compute_attenuation_viscoelastic.f90:36-236); returns the
// sums of e1, e11, e13 over the SLS.  w5i: 5 x warp + i of the point, so that
// the arrays are [warp][i][..][row].  Coefficients: Newmark {A1, A2, B1, B2},
// LDDRK {1/tau1, 1/tau2, phi1, phi2} per SLS, from the point's set or its own.
template <bool LDDRK, bool OWN>
__device__ __forceinline__ void attenuation_point(const Params &P, size_t w5i, int lane, int set, float dux_dxl,
                                                  float dux_dzl, float duz_dxl, float duz_dzl, int stage, float &e1s,
                                                  float &e11s, float &e13s) {
  float4 cc[3];
#pragma unroll
  for (int s = 0; s < 3; ++s) cc[s] = OWN ? __ldg(P.att_coef + w5i * 96 + 32 * s + lane) : __ldg(P.att_sets + 3 * set + s);
  const float theta_n = dux_dxl + duz_dzl;
  if (!LDDRK) {
    float4 *st = P.att_a + (w5i * 3) * 32 + lane;
    const float4 s0 = st[0], s1 = st[32], s2 = st[64];
    float e1[3] = {s0.x, s0.y, s0.z}, e11[3] = {s0.w, s1.x, s1.y}, e13[3] = {s1.z, s1.w, s2.x};
    const float old_xx = s2.y, old_zz = s2.z, old_xz = s2.w;
    const float theta_n1 = old_xx + old_zz;
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      float a = cc[s].x;
      e1[s] = a * a * e1[s] + cc[s].z * (theta_n + a * theta_n1);
      a = cc[s].y;
      e11[s] = a * a * e11[s] + cc[s].w * (dux_dxl - theta_n / 2.f + a * (old_xx - theta_n1 / 2.f));
      e13[s] = a * a * e13[s] + cc[s].w * (dux_dzl + duz_dxl + a * old_xz);
    }
    st[0] = make_float4(e1[0], e1[1], e1[2], e11[0]);
    st[32] = make_float4(e11[1], e11[2], e13[0], e13[1]);
    st[64] = make_float4(e13[2], dux_dxl, duz_dzl, dux_dzl + duz_dxl);
    e1s = e1[0] + e1[1] + e1[2];
    e11s = e11[0] + e11[1] + e11[2];
    e13s = e13[0] + e13[1] + e13[2];
  } else {
    float4 *st = P.att_a + (w5i * 2) * 32 + lane, *sl = P.att_al + (w5i * 2) * 32 + lane;
    float *tt = P.att_c + w5i * 32 + lane, *tl = P.att_cl + w5i * 32 + lane;
    const float4 s0 = st[0], s1 = st[32], l0 = sl[0], l1 = sl[32];
    float e[9] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w, *tt};
    float l[9] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w, *tl};
    const float al = P.alpha[stage], be = P.beta[stage];
    const double dt = static_cast<double>(P.dt);
    const float in[3] = {theta_n, dux_dxl - theta_n / 2.f, dux_dzl + duz_dxl};
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      // 1/tau_sigma is a double in the reference: these products are double there too
      const double itau = k < 3 ? cc[k % 3].x : cc[k % 3].y;
      const float phi = k < 3 ? cc[k % 3].z : cc[k % 3].w;
      if (k < 3)
        l[k] = static_cast<float>(static_cast<double>(al * l[k]) +
                                  dt * (static_cast<double>(in[0] * phi) - static_cast<double>(e[k]) * itau));
      else
        l[k] = static_cast<float>(static_cast<double>(al * l[k] + P.dt * (in[k / 3] * phi)) -
                                  dt * (static_cast<double>(e[k]) * itau));
      e[k] = e[k] + be * l[k];
    }
    st[0] = make_float4(e[0], e[1], e[2], e[3]);
    st[32] = make_float4(e[4], e[5], e[6], e[7]);
    *tt = e[8];
    sl[0] = make_float4(l[0], l[1], l[2], l[3]);
    sl[32] = make_float4(l[4], l[5], l[6], l[7]);
    *tl = l[8];
    e1s = e[0] + e[1] + e[2];
    e11s = e[3] + e[4] + e[5];
    e13s = e[6] + e[7] + e[8];
  }
}

// Sensitivity-kernel integrands at one element point (compute_kernels.f90:75-292):
// strains of the adjoint field and of the forward frame (b) with the mapping
// derivatives used in double, as the reference declares them.
__device__ __forceinline__ float2 kernel_point(float2 dxi, float2 dg, float2 bxi, float2 bg, float4 g) {
  const double xixl = g.x, xizl = g.y, gammaxl = g.z, gammazl = g.w;
  const float dux_dxl = static_cast<float>(dxi.x * xixl + dg.x * gammaxl);
  const float dux_dzl = static_cast<float>(dxi.x * xizl + dg.x * gammazl);
  const float duz_dxl = static_cast<float>(dxi.y * xixl + dg.y * gammaxl);
  const float duz_dzl = static_cast<float>(dxi.y * xizl + dg.y * gammazl);
  const float bdux_dxl = static_cast<float>(bxi.x * xixl + bg.x * gammaxl);
  const float bdux_dzl = static_cast<float>(bxi.x * xizl + bg.x * gammazl);
  const float bduz_dxl = static_cast<float>(bxi.y * xixl + bg.y * gammaxl);
  const float bduz_dzl = static_cast<float>(bxi.y * xizl + bg.y * gammazl);
  const float dsxz = static_cast<float>(0.5 * (static_cast<double>(duz_dxl) + static_cast<double>(dux_dzl)));
  const float bdsxz = static_cast<float>(0.5 * (static_cast<double>(bduz_dxl) + static_cast<double>(bdux_dzl)));
  const float kap = (dux_dxl + duz_dzl) * (bdux_dxl + bduz_dzl);
  return make_float2(kap, dux_dxl * bdux_dxl + duz_dzl * bduz_dzl + 2.f * dsxz * bdsxz - 1.f / 3.f * kap);
}

// Registers: as many CTAs as possible without spilling the row.  1000 x 400
// elements take 175, 173 and 178 us with 64, 80 and 96; an attenuating 800 x
// 400 mesh 264, 242 and 286 us with 80, 96 and 112; gradients gain 2 to 4 %
// from 96.
constexpr int row_regs(bool atten, bool kern) { return atten || kern ? 96 : 80; }

// OWN: every point reads coefficients of its own, 48 bytes that a warp reads in
// order.  Per step of 600 x 300 elements whose points draw their set at random,
// through the sets / OWN: 155 / 159 us with 192 sets, 162 / 159 with 3,072,
// 174 / 159 with 49,152, 192 / 159 where all points differ; 301 x 150 with LDDRK
// 434 / 456 us with 3,072, 451 / 456 with 49,152, 472 / 456 with 390,000 (where
// finding 49,152 sets takes 0.2 s more than a solver without).  A medium that is
// constant inside elements stays with the sets (148 us where all elements
// differ).
template <bool ANISO, bool ATTEN, bool LDDRK, bool KERN, bool OWN>
__global__ void __maxnreg__(row_regs(ATTEN, KERN))
    k_elastic_rows(const Params P, int record_prev, int stage, int tile0, int kstep) {
  extern __shared__ __align__(16) unsigned char smem[];
  const TileInfo &ti = P.tiles[tile0 + blockIdx.x];
  const int tid = threadIdx.x, NT = blockDim.x, lane = tid & 31;
  const int n_int = ti.n_int, nl = n_int + ti.n_sh, int_begin = ti.int_begin, sh_off = ti.sh_off, ncol = ti.ncol;
  const bool have = tid < 5 * ti.nelem;
  const int e = tid / 5, j = tid - 5 * e;
  const RowSmem L = row_smem_layout(P.max_local, P.max_elems, KERN);
  float2 *s_u = reinterpret_cast<float2 *>(smem);
  float2 *s_v = reinterpret_cast<float2 *>(smem + L.v);
  float2 *s_acc = reinterpret_cast<float2 *>(smem + L.acc);
  float2 *s_b = reinterpret_cast<float2 *>(smem + L.b);
  float2 *s_rm = reinterpret_cast<float2 *>(smem + L.rm);
  int *s_id = reinterpret_cast<int *>(smem + L.w);  // device points of the shared points, until phase 4
  float2 *s_w = reinterpret_cast<float2 *>(smem + L.w) + 25 * e;
  float2 *s_wb = reinterpret_cast<float2 *>(smem + L.wb) + 25 * e;
  float2 *s_t = reinterpret_cast<float2 *>(smem + L.t) + 25 * e;
  float *s_h = reinterpret_cast<float *>(smem + L.h);

  // every thread copies what it will use itself: no load of a point loop is waited for in the loop
  for (int l = n_int + tid; l < nl; l += NT) {
    cp_async4(s_id + l - n_int, P.sh_ids + sh_off + l - n_int);
    cp_async4(s_rm + l, P.sh_slot + sh_off + l - n_int);
  }
  cp_async_commit();
  // what does not change from step to step is requested before the previous
  // kernel is waited for
  const size_t wbase = static_cast<size_t>((ti.lane0 + tid) >> 5);
  float4 geo[5];
  float2 mat[5];
  uint32_t id[3];
  uint32_t phase = 0;
#pragma unroll
  for (int k = 0; k < 3; ++k) id[k] = 0;
  if (have) {
#pragma unroll
    for (int k = 0; k < 3; ++k) id[k] = __ldg(P.rid + (wbase * 3 + k) * 32 + lane);
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      geo[i] = __ldg(P.rgeo + (wbase * 5 + i) * 32 + lane);
      mat[i] = __ldg(P.rmat + (wbase * 5 + i) * 32 + lane);
    }
    phase = __ldg(P.rphase + ti.elem_base + e);
  }
  // what is read and written in place goes to L2 meanwhile
  if (lane == 0 && (tid & ~31) < 5 * ti.nelem) {
    if (ATTEN) prefetch_l2(P.att_a + wbase * 5 * (LDDRK ? 2 : 3) * 32, 5 * (LDDRK ? 2 : 3) * 32 * sizeof(float4));
    if (OWN) prefetch_l2(P.att_coef + wbase * 5 * 96, 5 * 96 * sizeof(float4));
    if (ATTEN && LDDRK) {
      prefetch_l2(P.att_al + wbase * 5 * 2 * 32, 5 * 2 * 32 * sizeof(float4));
      prefetch_l2(P.att_c + wbase * 5 * 32, 5 * 32 * sizeof(float));
      prefetch_l2(P.att_cl + wbase * 5 * 32, 5 * 32 * sizeof(float));
    }
    if (KERN) prefetch_l2(P.kmu_kl + wbase * 5 * 32, 5 * 32 * sizeof(float2));
    if (tid == 0 && LDDRK) {
      prefetch_l2(P.vL + int_begin, n_int * sizeof(float2));
      prefetch_l2(P.uL + int_begin, n_int * sizeof(float2));
    }
    if (tid == 0 && KERN) prefetch_l2(P.rho_kl_glob + int_begin, n_int * sizeof(float));
  }
  for (int k = tid; k < 60; k += NT) s_h[k] = k < 55 ? P.hconst[k < 50 ? k : k + 5] : P.hsum[k - 55];

  for (int l = tid; l < n_int; l += NT) cp_async8(s_rm + l, P.rmass + int_begin + l);
  cp_async_commit();
  wait_previous_kernel();
  const int step = *P.d_step + kstep;
  // receivers of the previous step read the old fields before any write
  if (record_prev)
    for (int r = tid; r < ti.rec_n; r += NT) record_receiver(P, ti.rec_off + r, step - 1);
  // a masked member neither reads nor writes its points from here on (uniform over the CTA)
  if (P.tile_member && P.member_status[P.tile_member[tile0 + blockIdx.x]]) {
    cp_async_wait_all();
    return;
  }
  const float2 *kframe = nullptr;
  if (KERN) kframe = P.kframes + static_cast<size_t>(*P.kern_base - step) * P.nglob;

  // 1. every field load of the tile is issued at once, straight into shared memory
  auto fetch = [&](int l, int g) {
    cp_async8(s_u + l, P.u + g);
    cp_async8(s_v + l, P.v + g);
    if (!LDDRK) cp_async8(s_acc + l, P.a + g);
    if (KERN) cp_async8(s_b + l, kframe + g);
  };
  for (int l = tid; l < n_int; l += NT) fetch(l, int_begin + l);
  cp_async_commit();
  cp_async_wait<2>();  // the shared points' ids
  for (int l = n_int + tid; l < nl; l += NT) fetch(l, s_id[l - n_int]);
  cp_async_wait_all();
  __syncthreads();

  // 2. Newmark predictor in place (the interior points' displacement goes out),
  //    or a cleared accumulator for an LDDRK stage
  const float dt = P.dt, dto2 = P.dto2, dt2o2 = P.dt2o2;
  int frame = -1;
  if (P.frames) {
    const int fi = step - *P.frame_base;
    if (fi >= 0 && fi < P.nframes) frame = fi;
  }
  bool bad = false;
  for (int l = tid; l < nl; l += NT) {
    if (!LDDRK) {
      float2 u = s_u[l], v = s_v[l];
      const float2 a = s_acc[l];
      u.x = newmark_displ(u.x, v.x, a.x, dt, dt2o2);
      u.y = newmark_displ(u.y, v.y, a.y, dt, dt2o2);
      v.x = newmark_veloc(v.x, a.x, dto2);
      v.y = newmark_veloc(v.y, a.y, dto2);
      s_u[l] = u;
      s_v[l] = v;
      if (l < n_int) {
        P.u[int_begin + l] = u;
        if (frame >= 0) P.frames[static_cast<size_t>(frame) * P.nglob + int_begin + l] = u;
        bad |= !(fabsf(u.x) < 1e25f && fabsf(u.y) < 1e25f);
      }
    }
    s_acc[l] = make_float2(0.f, 0.f);
  }
  __syncthreads();
  // outer edge of a CPML layer: displacement and velocity zeroed before the
  // forces (pml_boundary_elastic, pml_compute.f90:545-574)
  if (ti.edge_n > 0) {
    for (int k = tid; k < ti.edge_n; k += NT) {
      const int l = P.edge_local[ti.edge_off + k];
      s_u[l] = make_float2(0.f, 0.f);
      s_v[l] = make_float2(0.f, 0.f);
      if (!LDDRK && l < n_int) {
        P.u[int_begin + l] = make_float2(0.f, 0.f);
        if (frame >= 0) P.frames[static_cast<size_t>(frame) * P.nglob + int_begin + l] = make_float2(0.f, 0.f);
      }
    }
    __syncthreads();
  }

  // 3. boundary terms, coupling and sources (element terms follow after a barrier)
  boundary_terms(P, ti, s_v, s_acc, step, stage, tid, NT);

  // 4. the element rows
  const uint32_t lid[5] = {id[0] & 0xffffu, id[0] >> 16, id[1] & 0xffffu, id[1] >> 16, id[2] & 0xffffu};
  float2 w[5], uc = make_float2(0.f, 0.f), wb[5], bc = uc;
  if (have) {
    uc = s_u[id[2] >> 16];
    if (KERN) bc = s_b[id[2] >> 16];
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      w[i] = f2_sub(s_u[lid[i]], uc);
      s_w[5 * j + i] = w[i];
      if (KERN) {
        wb[i] = f2_sub(s_b[lid[i]], bc);
        s_wb[5 * j + i] = wb[i];
      }
    }
  }
  __syncthreads();
  float2 r[5];
  if (have) {
    float2 dxi[5], dg[5], bxi[5], bg[5];
    row_derivs(P, w, uc, dxi);
    if (KERN) row_derivs(P, wb, bc, bxi);
    const float hs = s_h[55 + j];
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      dg[i] = make_float2(uc.x * hs, uc.y * hs);
      if (KERN) bg[i] = make_float2(bc.x * hs, bc.y * hs);
    }
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const float2 h = make_float2(s_h[5 * j + k], s_h[5 * j + k]);
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        dg[i] = f2_fma2(s_w[5 * k + i], h, dg[i]);
        if (KERN) bg[i] = f2_fma2(s_wb[5 * k + i], h, bg[i]);
      }
    }
    int aset = 0, arow = -1;
    if (ATTEN && !OWN && P.att_eset) aset = __ldg(P.att_eset + ti.elem_base + e);
    if (ANISO && (phase >> 31)) arow = __ldg(P.rani + ti.elem_base + e);
    float2 t1[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      const float4 g4 = geo[i];
      if (KERN) {
        float2 *km = P.kmu_kl + (wbase * 5 + i) * 32 + lane;
        const float2 a = kernel_point(dxi[i], dg[i], bxi[i], bg[i], g4), o = *km;
        *km = make_float2(o.x + a.x, o.y + a.y);
      }
      const float dux_dxl = dxi[i].x * g4.x + dg[i].x * g4.z;
      const float dux_dzl = dxi[i].x * g4.y + dg[i].x * g4.w;
      const float duz_dxl = dxi[i].y * g4.x + dg[i].y * g4.z;
      const float duz_dzl = dxi[i].y * g4.y + dg[i].y * g4.w;
      const float jac = 1.f / (g4.x * g4.w - g4.z * g4.y);
      const float lam = mat[i].x, mu = mat[i].y;
      const float lp2m = lam + 2.f * mu;
      float sxx = lp2m * dux_dxl + lam * duz_dzl;
      float szz = lp2m * duz_dzl + lam * dux_dxl;
      float sxz = mu * (duz_dxl + dux_dzl);
      if (ANISO && arow >= 0) {  // stress in double (compute_forces_viscoelastic.F90:372-445)
        const size_t ap = static_cast<size_t>(arow) * 25 + 5 * j + i;
        const float4 ca = __ldg(P.rc4 + ap);
        const float2 cb = __ldg(P.rc2 + ap);
        const double c11 = ca.x, c13 = ca.y, c15 = ca.z, c33 = ca.w, c35 = cb.x, c55 = cb.y;
        const double sh = static_cast<double>(duz_dxl) + static_cast<double>(dux_dzl);
        sxx = static_cast<float>(c11 * dux_dxl + c13 * duz_dzl + c15 * sh);
        szz = static_cast<float>(c13 * dux_dxl + c33 * duz_dzl + c35 * sh);
        sxz = static_cast<float>(c15 * dux_dxl + c35 * duz_dzl + c55 * sh);
      }
      if (ATTEN) {
        if (!OWN && P.att_pset) aset = __ldg(P.att_pset + (wbase * 5 + i) * 32 + lane);
        float e1s, e11s, e13s;
        attenuation_point<LDDRK, OWN>(P, wbase * 5 + i, lane, aset, dux_dxl, dux_dzl, duz_dxl, duz_dzl, stage, e1s, e11s, e13s);
        sxx = sxx + (lam + mu) * e1s + 2.f * mu * e11s;
        sxz = sxz + mu * e13s;
        szz = szz + (lam + mu) * e1s - 2.f * mu * e11s;
      }
      t1[i] = make_float2(jac * (sxx * g4.x + sxz * g4.y), jac * (sxz * g4.x + szz * g4.y));
      s_t[5 * j + i] = make_float2(jac * (sxx * g4.z + sxz * g4.w), jac * (sxz * g4.z + szz * g4.w));
    }
    row_transposed(P, t1, r);
  }
  __syncthreads();
  if (have) {
    float2 col[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const float h = s_h[25 + 5 * k + j];
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        const float2 t = s_t[5 * k + i];
        col[i] = k == 0 ? make_float2(t.x * h, t.y * h) : f2_fma2(t, make_float2(h, h), col[i]);
      }
    }
    const float wz = s_h[50 + j];
#pragma unroll
    for (int i = 0; i < 5; ++i)
      r[i] = f2_fma(col[i], P.hconst[50 + i], make_float2(wz * r[i].x, wz * r[i].y));
  }

  // 5. assembly: no two threads add to one point in one phase.  A row's first
  //    four points are of class 0 or 2, its last one of class 1 or 3
  const int pa = (phase >> (j == 4 ? 16 : 0)) & 127, pb = (phase >> (j == 4 ? 24 : 8)) & 127;
  for (int p = 0; p < ncol; ++p) {
    if (have && pa == p) {
#pragma unroll
      for (int i = 0; i < 4; ++i) r[i] = f2_sub(s_acc[lid[i]], r[i]);
#pragma unroll
      for (int i = 0; i < 4; ++i) s_acc[lid[i]] = r[i];
    }
    if (have && pb == p) s_acc[lid[4]] = f2_sub(s_acc[lid[4]], r[4]);
    __syncthreads();
  }

  // 6. mass matrix, corrector or LDDRK update, write-back
  for (int l = tid; l < nl; l += NT) {
    const float2 acc = s_acc[l], rm = s_rm[l];
    if (l >= n_int) {
      P.partial[__float_as_int(rm.x)] = acc;
      continue;
    }
    const int g = int_begin + l;
    const float2 a = make_float2(acc.x * rm.x, acc.y * rm.y);
    float2 v = s_v[l];
    if (!LDDRK) {
      v.x = v.x + dto2 * a.x;
      v.y = v.y + dto2 * a.y;
    } else {
      const float al = P.alpha[stage], be = P.beta[stage];
      float2 u = s_u[l], vl = P.vL[g], ul = P.uL[g];
      vl.x = al * vl.x + dt * a.x;
      vl.y = al * vl.y + dt * a.y;
      ul.x = al * ul.x + dt * v.x;
      ul.y = al * ul.y + dt * v.y;
      v.x = v.x + be * vl.x;
      v.y = v.y + be * vl.y;
      u.x = u.x + be * ul.x;
      u.y = u.y + be * ul.y;
      P.vL[g] = vl;
      P.uL[g] = ul;
      P.u[g] = u;
      if (frame >= 0) P.frames[static_cast<size_t>(frame) * P.nglob + g] = u;
      bad |= !(fabsf(u.x) < 1e25f && fabsf(u.y) < 1e25f);
    }
    P.v[g] = v;
    P.a[g] = a;
    if (frame >= 0 && P.aframes) P.aframes[static_cast<size_t>(frame) * P.nglob + g] = a;
    if (KERN) {
      const float2 b = s_b[l];
      P.rho_kl_glob[g] = P.rho_kl_glob[g] + (a.x * b.x + a.y * b.y);
      if (P.hess_glob) {
        // compute_kernels_Hessian: |b_accel|^2 and accel . b_accel at the point
        const float2 ba = P.kaframes[static_cast<size_t>(*P.kern_base - step) * P.nglob + g];
        float2 h = P.hess_glob[g];
        h.x = h.x + (ba.x * ba.x + ba.y * ba.y);
        h.y = h.y + (a.x * ba.x + a.y * ba.y);
        P.hess_glob[g] = h;
      }
    }
  }
  if (bad) {
    if (P.tile_member)
      P.member_status[P.tile_member[tile0 + blockIdx.x]] = 1;
    else
      *P.d_status = 1;
  }
}

}  // namespace sf2d

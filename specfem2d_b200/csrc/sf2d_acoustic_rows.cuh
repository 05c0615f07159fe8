// Tile kernel of the fluid with one element row per thread: the scalar
// counterpart of sf2d_rows.cuh, whose remarks on the split, the prefetches and
// the differences to the element's centre hold here too.
// Against tasks of rows, columns and points, a run with a fluid of 400 x 80
// elements under CPML takes 6.15 ms instead of 6.67 and a gradient over a
// 250 x 100 element ocean model 13.3 ms instead of 16.6; one element per thread
// was slower (7.15 and 16.6 ms).
#pragma once

#include "sf2d_acoustic.cuh"

namespace sf2d {

// Shared memory of a tile by rows: chi, chi_dot, accumulator, inverse mass or
// partial-sum slot (and the forward frame) and mask of its points; per element
// 25 differences to the centre (and the frame's) and 25 gamma terms; the line
// matrices.
struct AcRowSmem {
  size_t pd, acc, rm, b, w, wb, t, h, mask, total;
};
__host__ __device__ inline AcRowSmem ac_row_smem_layout(int max_local, int max_elems, bool kern) {
  const size_t lb = align16(static_cast<size_t>(max_local) * sizeof(float));
  const size_t eb = align16(static_cast<size_t>(max_elems) * 25 * sizeof(float));
  AcRowSmem L;
  L.pd = lb;
  L.acc = 2 * lb;
  L.rm = 3 * lb;
  L.b = 4 * lb;
  L.w = L.b + (kern ? lb : 0);
  L.wb = L.w + eb;
  L.t = L.wb + (kern ? eb : 0);
  L.h = L.t + eb;
  L.mask = L.h + 64 * sizeof(float);
  L.total = align16(L.mask + static_cast<size_t>(max_local));
  return L;
}

__device__ __forceinline__ void ac_row_derivs(const AcParams &A, const float (&w)[5], float pc, float (&out)[5]) {
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    float d = pc * A.hsum[m];
#pragma unroll
    for (int k = 0; k < 5; ++k) d = fmaf(w[k], A.hconst[5 * m + k], d);
    out[m] = d;
  }
}

constexpr int AC_ROW_REGS = 72;  // the smallest count without spills

// KERN: an adjoint run that accumulates the fluid kernels
// (compute_kernels.f90:293-449): grad(chi_adj) . grad(chi) per element point,
// chi_adj_dd chi per fluid point; 1/rho, 1/kappa and dt follow when the sums
// are read.
template <bool LDDRK, bool KERN>
__global__ void __maxnreg__(AC_ROW_REGS) k_acoustic_rows(const AcParams A, int stage, int tile0, int kstep) {
  extern __shared__ __align__(16) unsigned char smem[];
  const TileInfo &ti = A.tiles[tile0 + blockIdx.x];
  const int tid = threadIdx.x, NT = blockDim.x, lane = tid & 31;
  const int n_int = ti.n_int, nl = n_int + ti.n_sh, int_begin = ti.int_begin, sh_off = ti.sh_off, ncol = ti.ncol;
  const bool have = tid < 5 * ti.nelem;
  const int e = tid / 5, j = tid - 5 * e;
  const AcRowSmem L = ac_row_smem_layout(A.max_local_l, A.max_elems_l, KERN);
  float *s_p = reinterpret_cast<float *>(smem);
  float *s_pd = reinterpret_cast<float *>(smem + L.pd);
  float *s_acc = reinterpret_cast<float *>(smem + L.acc);
  float *s_rm = reinterpret_cast<float *>(smem + L.rm);
  float *s_b = reinterpret_cast<float *>(smem + L.b);
  int *s_id = reinterpret_cast<int *>(smem + L.w);  // device points of the shared points, until phase 4
  float *s_w = reinterpret_cast<float *>(smem + L.w) + 25 * e;
  float *s_wb = reinterpret_cast<float *>(smem + L.wb) + 25 * e;
  float *s_t = reinterpret_cast<float *>(smem + L.t) + 25 * e;
  float *s_h = reinterpret_cast<float *>(smem + L.h);
  uint8_t *s_mask = reinterpret_cast<uint8_t *>(smem + L.mask);

  // every thread copies what it will use itself: no load of a point loop is waited for in the loop
  for (int l = n_int + tid; l < nl; l += NT) {
    cp_async4(s_id + l - n_int, A.sh_ids + sh_off + l - n_int);
    cp_async4(s_rm + l, A.sh_slot + sh_off + l - n_int);
  }
  cp_async_commit();
  const size_t wbase = static_cast<size_t>((ti.lane0 + tid) >> 5);
  float4 geo[5];
  float fac[5];
  uint32_t id[3] = {0, 0, 0};
  uint32_t phase = 0;
  if (have) {
#pragma unroll
    for (int k = 0; k < 3; ++k) id[k] = __ldg(A.lid + (wbase * 3 + k) * 32 + lane);
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      const size_t o = (wbase * 5 + i) * 32 + lane;
      geo[i] = __ldg(A.lgeo + o);
      fac[i] = __ldg(A.lfac + o);
    }
    phase = __ldg(A.lphase + ti.elem_base + e);
  }
  for (int l = tid; l < n_int; l += NT) cp_async4(s_rm + l, A.rmass + int_begin + l);
  cp_async_commit();
  for (int k = tid; k < 60; k += NT) s_h[k] = k < 55 ? A.hconst[k < 50 ? k : k + 5] : A.hsum[k - 55];
  wait_previous_kernel();
  // fluid receivers are recorded by k_acoustic_receivers after each step: their
  // double-precision gradient would hold registers through the whole tile
  const int step = *A.d_step + kstep;
  int frame = -1;
  if (A.pframes) {
    const int fi = step - *A.pframe_base;
    if (fi >= 0 && fi < A.npframes) frame = fi;
  }
  const float *kframe = nullptr;
  if (KERN) {
    const int fi = *A.kp_base - step;
    if (fi >= 0 && fi < A.npframes) kframe = A.kpframes + static_cast<size_t>(fi) * A.nglob_ac;
  }

  // 1. loads
  auto fetch = [&](int l, int g) {
    cp_async4(s_p + l, A.p + g);
    cp_async4(s_pd + l, A.pd + g);
    if (!LDDRK) cp_async4(s_acc + l, A.pdd + g);
    if (KERN && kframe) cp_async4(s_b + l, kframe + g);
  };
  for (int l = tid; l < n_int; l += NT) fetch(l, int_begin + l);
  cp_async_commit();
  cp_async_wait<2>();  // the shared points' ids
  for (int l = n_int + tid; l < nl; l += NT) fetch(l, s_id[l - n_int]);
  cp_async_wait_all();
  __syncthreads();

  // 2. predictor (or cleared accumulator); the interior points' chi is final
  //    with Newmark and goes out
  const float dt = A.dt, dto2 = A.dto2, dt2o2 = A.dt2o2;
  bool bad = false;
  auto put_p = [&](int g, float p) {
    A.p[g] = p;
    if (frame >= 0) A.pframes[static_cast<size_t>(frame) * A.nglob_ac + g] = p;
    bad |= !(fabsf(p) < 1e25f);
  };
  for (int l = tid; l < nl; l += NT) {
    if (!LDDRK) {
      const float pdd = s_acc[l], pd = s_pd[l], p = newmark_displ(s_p[l], pd, pdd, dt, dt2o2);
      s_p[l] = p;
      s_pd[l] = newmark_veloc(pd, pdd, dto2);
      if (l < n_int) put_p(int_begin + l, p);
    }
    s_acc[l] = 0.f;
    s_mask[l] = 0;
  }
  __syncthreads();
  // free-surface and layer-edge points, zeroed and flagged for step 6
  if (ti.edge_n > 0) {
    for (int k = tid; k < ti.edge_n; k += NT) {
      const int v = A.edge_local[ti.edge_off + k], l = v & 0xFFFF;
      s_p[l] = 0.f;
      s_pd[l] = 0.f;
      s_mask[l] = static_cast<uint8_t>(v >> 16);
      if (!LDDRK && l < n_int) put_p(int_begin + l, 0.f);
    }
    __syncthreads();
  }

  // 3. boundary terms, coupling and sources
  ac_boundary_terms<LDDRK>(A, ti, s_pd, s_acc, step, stage, tid, NT);

  // 4. the element rows
  const uint32_t lid[5] = {id[0] & 0xffffu, id[0] >> 16, id[1] & 0xffffu, id[1] >> 16, id[2] & 0xffffu};
  float w[5], pc = 0.f, wb[5], bc = 0.f;
  if (have) {
    pc = s_p[id[2] >> 16];
    if (KERN && kframe) bc = s_b[id[2] >> 16];
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      w[i] = s_p[lid[i]] - pc;
      s_w[5 * j + i] = w[i];
      if (KERN && kframe) {
        wb[i] = s_b[lid[i]] - bc;
        s_wb[5 * j + i] = wb[i];
      }
    }
  }
  __syncthreads();
  float r[5];
  if (have) {
    float dxi[5], dg[5];
    ac_row_derivs(A, w, pc, dxi);
    const float hs = s_h[55 + j];
#pragma unroll
    for (int i = 0; i < 5; ++i) dg[i] = pc * hs;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const float h = s_h[5 * j + k];
#pragma unroll
      for (int i = 0; i < 5; ++i) dg[i] = fmaf(s_w[5 * k + i], h, dg[i]);
    }
    if (KERN && kframe) {
      float bxi[5], bg[5];
      ac_row_derivs(A, wb, bc, bxi);
#pragma unroll
      for (int i = 0; i < 5; ++i) bg[i] = bc * hs;
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        const float h = s_h[5 * j + k];
#pragma unroll
        for (int i = 0; i < 5; ++i) bg[i] = fmaf(s_wb[5 * k + i], h, bg[i]);
      }
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        // the mapping applied in double and stored in FP32, as the reference does
        const size_t o = (wbase * 5 + i) * 32 + lane;
        const float4 g = geo[i];
        const float ax = static_cast<float>(static_cast<double>(dxi[i]) * g.x + static_cast<double>(dg[i]) * g.z);
        const float az = static_cast<float>(static_cast<double>(dxi[i]) * g.y + static_cast<double>(dg[i]) * g.w);
        const float bx = static_cast<float>(static_cast<double>(bxi[i]) * g.x + static_cast<double>(bg[i]) * g.z);
        const float bz = static_cast<float>(static_cast<double>(bxi[i]) * g.y + static_cast<double>(bg[i]) * g.w);
        A.kl_ac[o] = A.kl_ac[o] + (ax * bx + az * bz);
      }
    }
    float t1[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      const float4 g = geo[i];
      const float dx = dxi[i] * g.x + dg[i] * g.z, dz = dxi[i] * g.y + dg[i] * g.w;
      t1[i] = fac[i] * (g.x * dx + g.y * dz);
      s_t[5 * j + i] = fac[i] * (g.z * dx + g.w * dz);
    }
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      float d = t1[0] * A.hconst[25 + m];
#pragma unroll
      for (int k = 1; k < 5; ++k) d = fmaf(t1[k], A.hconst[25 + 5 * k + m], d);
      r[m] = d;
    }
  }
  __syncthreads();
  if (have) {
    float col[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const float h = s_h[25 + 5 * k + j];
#pragma unroll
      for (int i = 0; i < 5; ++i) col[i] = k == 0 ? s_t[i] * h : fmaf(s_t[5 * k + i], h, col[i]);
    }
    const float wz = s_h[50 + j];
#pragma unroll
    for (int i = 0; i < 5; ++i) r[i] = wz * r[i] + A.hconst[50 + i] * col[i];
  }

  // 5. assembly: no two threads add to one point in one phase
  const int pa = (phase >> (j == 4 ? 16 : 0)) & 127, pb = (phase >> (j == 4 ? 24 : 8)) & 127;
  for (int p = 0; p < ncol; ++p) {
    if (have && pa == p) {
#pragma unroll
      for (int i = 0; i < 4; ++i) r[i] = s_acc[lid[i]] - r[i];
#pragma unroll
      for (int i = 0; i < 4; ++i) s_acc[lid[i]] = r[i];
    }
    if (have && pb == p) s_acc[lid[4]] = s_acc[lid[4]] - r[4];
    __syncthreads();
  }

  // 6. mass, corrector or LDDRK update, free surface, write-back
  for (int l = tid; l < nl; l += NT) {
    const float acc = s_acc[l], rm = s_rm[l];
    if (l >= n_int) {
      A.partial[__float_as_int(rm)] = acc;
      continue;
    }
    const int g = int_begin + l;
    float pdd = acc * rm;
    float pd = s_pd[l], p = s_p[l];
    if (!LDDRK) {
      pd = newmark_veloc(pd, pdd, dto2);
    } else {
      const float al = A.alpha[stage], be = A.beta[stage];
      float pdl = A.pdL[g], pl = A.pL[g];
      pdl = al * pdl + dt * pdd;
      pl = al * pl + dt * pd;
      pd = pd + be * pdl;
      p = p + be * pl;
      A.pdL[g] = pdl;
      A.pL[g] = pl;
    }
    if (s_mask[l]) {
      p = 0.f;
      pd = 0.f;
      pdd = 0.f;
    }
    if (LDDRK) put_p(g, p);
    A.pd[g] = pd;
    A.pdd[g] = pdd;
    if (KERN && kframe) A.kap_glob[g] = A.kap_glob[g] + pdd * s_b[l];
  }
  if (bad) *A.d_status = 1;
}

// Fluid kernel sums to element order: rho' = dt / rho sum, kappa' = dt / kappa
// sum (one thread per element point; lane: first row of each element).
static __global__ void k_fluid_kernels(const float *kl, const float *kap_glob, const int *lane, const int *point,
                                       const float2 *rk, float dt, int n, float *out) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int q = p % 25, r = lane[p / 25] + q / 5;
  const float2 m = rk[p];
  out[p] = 1.f / m.x * kl[(static_cast<size_t>(r >> 5) * 5 + q % 5) * 32 + (r & 31)] * dt;
  out[n + p] = 1.f / m.y * kap_glob[point[p]] * dt;
}

}  // namespace sf2d

// Host-side solver object shared by the C-ABI translation units.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "sf2d_b200.h"
#include "sf2d_kernels.cuh"
#include "sf2d_rows.cuh"
#include "sf2d_tiler.h"

namespace sf2d {
// Sets the calling thread's last error message and returns `code`.
int fail(int code, const std::string &msg);
const char *last_error();
}  // namespace sf2d

using sf2d::fail;

#define SF2D_CUDA(call)                                                                       \
  do {                                                                                        \
    cudaError_t e_ = (call);                                                                  \
    if (e_ != cudaSuccess)                                                                    \
      return fail(e_ == cudaErrorMemoryAllocation ? SF2D_ERR_OOM : SF2D_ERR_CUDA,             \
                  std::string(#call) + ": " + cudaGetErrorString(e_));                        \
  } while (0)

namespace sf2d {

// A step kernel with programmatic dependent launch: its CTAs may be scheduled
// while the kernel before it in the stream drains (every kernel launched so
// waits for its predecessor's completion before reading, wait_previous_kernel).
template <typename F, typename... A>
void launch_pdl(cudaStream_t stream, cudaError_t &first_error, F fn, int grid, int block, size_t smem_bytes, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(static_cast<unsigned>(block));
  cfg.dynamicSmemBytes = smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, fn, args...);
  if (e != cudaSuccess && first_error == cudaSuccess) first_error = e;
}

using TileKernel = void (*)(Params, int, int, int, int);

// Five threads an element and at most 96 registers a thread: 128 elements fit
// a CTA and the register file.
constexpr int MAX_ROW_ELEMS = 128;
constexpr size_t MAX_TILE_SMEM = 220 * 1024;

// A description's tile_elems: > 0 as given; -n "up to n"; 0 up to `standard`.
inline int tile_hint(int asked, int standard) {
  if (asked < 0) return -std::max(asked, -256);
  return asked > 0 ? asked : standard;
}

inline int sm_count() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 148;
  return n;
}

// Elements per tile by rows of a mesh (or domain) of n elements.  A size that
// is asked for is used; "up to" is halved (to 8 at least) while the tiles would
// not give every SM one and every other SM a second.  A step of a small mesh
// takes as long as one tile does: 80 x 60 elements take 9.9 us with 150 tiles of
// 32 and 8.8 us with 300 of 16; 233 x 147 elements (1071 tiles of 32) 17.9 us,
// and 19.1 us in tiles of 16.  Up to 32 elements stay in one tile, which needs no
// kernel for shared points: 3 x 3 elements 7.8 us, and 9.0 in tiles of 8; 6 x 5
// 7.8 and 8.9; 8 x 8 8.8 and 8.3.
inline int row_tile_elems(int asked, int standard, int n) {
  int te = std::min(tile_hint(asked, standard), MAX_ROW_ELEMS);
  if (asked > 0 || n <= std::min(te, 32)) return te;
  const long long sms = sm_count();
  while (te >= 16 && 2 * static_cast<long long>((n + te - 1) / te) < 3 * sms) te /= 2;
  return te;
}

template <bool ANISO, bool ATTEN, bool OWN>
inline TileKernel pick_rows_kernel(bool lddrk, bool kern) {
  if (kern) return k_elastic_rows<ANISO, ATTEN, false, true, OWN>;  // Newmark
  return lddrk ? k_elastic_rows<ANISO, ATTEN, true, false, OWN> : k_elastic_rows<ANISO, ATTEN, false, false, OWN>;
}
// own: every point has attenuation coefficients of its own
inline TileKernel pick_rows_kernel(bool aniso, bool atten, bool own, bool lddrk, bool kern) {
  if (aniso) {
    if (!atten) return pick_rows_kernel<true, false, false>(lddrk, kern);
    return own ? pick_rows_kernel<true, true, true>(lddrk, kern) : pick_rows_kernel<true, true, false>(lddrk, kern);
  }
  if (!atten) return pick_rows_kernel<false, false, false>(lddrk, kern);
  return own ? pick_rows_kernel<false, true, true>(lddrk, kern) : pick_rows_kernel<false, true, false>(lddrk, kern);
}

// the kernel of a CPML layer's tiles (isotropic, forward); visco: some layer
// elements attenuate (Newmark only)
template <int NT>
inline TileKernel pick_pml_kernel(bool lddrk, bool visco) {
  if (visco) return k_elastic_pml_tile<NT, true, false>;
  return lddrk ? k_elastic_pml_tile<NT, false, true> : k_elastic_pml_tile<NT, false, false>;
}
inline TileKernel pick_pml_kernel(int nt, bool lddrk, bool visco = false) {
  switch (nt) {
    case 128: return pick_pml_kernel<128>(lddrk, visco);
    case 250: return pick_pml_kernel<250>(lddrk, visco);
    case 512: return pick_pml_kernel<512>(lddrk, visco);
    default: return pick_pml_kernel<256>(lddrk, visco);
  }
}

// Boundary terms of each tile grouped by receiving point, so that one thread
// per point applies them (in parallel over points, in the reference's order at
// each point: Stacey, coupling, sources).  groups: one int4 per point (local
// point, first index into idx, Stacey count | coupling count << 8, source
// count); idx: the point's entries of each type in their list order.  The
// *_local vectors give each entry's tile-local point; tiles' st/cpl/src
// ranges index them.  Sets grp_off / grp_n of every tile.
inline std::string build_boundary_groups(std::vector<TileInfo> &tiles, const std::vector<int> &st_local,
                                         const std::vector<int> &cpl_local, const std::vector<int> &src_local,
                                         std::vector<int4> &groups, std::vector<int> &idx) {
  groups.clear();
  idx.clear();
  std::vector<std::vector<int>> st, cp, sr;
  std::vector<int> pts;
  for (TileInfo &t : tiles) {
    t.grp_off = static_cast<int>(groups.size());
    pts.clear();
    auto add = [&](std::vector<std::vector<int>> &lists, int l, int k) {
      if (static_cast<int>(st.size()) <= l) {
        st.resize(l + 1);
        cp.resize(l + 1);
        sr.resize(l + 1);
      }
      if (st[l].empty() && cp[l].empty() && sr[l].empty()) pts.push_back(l);
      lists[l].push_back(k);
    };
    for (int k = t.st_off; k < t.st_off + t.st_n; ++k) add(st, st_local[k], k);
    for (int k = t.cpl_off; k < t.cpl_off + t.cpl_n; ++k) add(cp, cpl_local[k], k);
    for (int k = t.src_off; k < t.src_off + t.src_n; ++k) add(sr, src_local[k], k);
    std::sort(pts.begin(), pts.end());
    for (int l : pts) {
      if (st[l].size() > 255 || cp[l].size() > 255) return "more than 255 boundary entries at one point";
      groups.push_back(make_int4(l, static_cast<int>(idx.size()),
                                 static_cast<int>(st[l].size() | (cp[l].size() << 8)), static_cast<int>(sr[l].size())));
      for (int k : st[l]) idx.push_back(k);
      for (int k : cp[l]) idx.push_back(k);
      for (int k : sr[l]) idx.push_back(k);
      st[l].clear();
      cp[l].clear();
      sr[l].clear();
    }
    t.grp_n = static_cast<int>(groups.size()) - t.grp_off;
  }
  return "";
}

}  // namespace sf2d

struct sf2d_solver {
  sf2d::Params P{};
  sf2d::Tiling T;
  std::vector<void *> allocs;
  int *d_dev2glob = nullptr;
  float2 *d_stage = nullptr;
  unsigned int *d_norm = nullptr;
  cudaStream_t stream = nullptr;
  size_t smem = 0;
  size_t dev_bytes = 0;
  int nglob = 0, nrec = 0, nstep_total = 0;
  int steps_done = 0;
  int chunk = 32;
  cudaGraphExec_t graph = nullptr;
  int graph_steps = 0;
  int nt = 256;      // threads per CTA asked for (the CPML tiles' default)
  int lane_nt = 32;  // threads per CTA of the tiles by rows: five per element of the largest, in whole warps
  // tiles by rows: slot -> the element's first row
  std::vector<int> slot_lane;
  // index of an element point in the blocks' [q][element] arrays
  size_t lane_index(int slot, int q) const {
    const int r = slot_lane[slot] + q / 5;
    return (static_cast<size_t>(r / 32) * 5 + q % 5) * 32 + r % 32;
  }
  unsigned char *att_buf = nullptr;  // every memory variable of the tiles by rows
  size_t att_bytes = 0;
  int pml_nt = 256, pml_max_q = 0, pml_max_local = 0;  // the CPML tiles' kernel
  int late_tile0 = 0;  // tiles [late_tile0, pml_tile0) touch points another domain uses
  int nmembers = 0;    // members of a packed batch (sf2d_set_members), 0 = none
  int priority = 0;    // of the solver's streams (0: the default, lowest)

  template <typename T_>
  int alloc(T_ **p, size_t count) {
    const size_t bytes = std::max<size_t>(count, 1) * sizeof(T_);
    cudaError_t e = cudaMalloc(reinterpret_cast<void **>(p), bytes);
    if (e != cudaSuccess)
      return fail(e == cudaErrorMemoryAllocation ? SF2D_ERR_OOM : SF2D_ERR_CUDA,
                  std::string("cudaMalloc: ") + cudaGetErrorString(e));
    allocs.push_back(*p);
    dev_bytes += bytes;
    return SF2D_OK;
  }
  template <typename T_>
  int upload(T_ **p, const T_ *host, size_t count) {
    int rc = alloc(p, count);
    if (rc) return rc;
    if (count) SF2D_CUDA(cudaMemcpy(*p, host, count * sizeof(T_), cudaMemcpyHostToDevice));
    return SF2D_OK;
  }
  using TileFn = void (*)(sf2d::Params, int, int, int, int);
  TileFn tile_fn = nullptr;
  TileFn pml_fn = nullptr;   // tiles [pml_tile0, ntiles) hold the CPML layer's elements
  int pml_tile0 = 0;
  size_t pml_smem = 0;
  size_t npml_q = 0;         // GLL points of the layer's elements
  bool lddrk = false;
  bool kern = false;
  bool atten = false;
  int nstage = 1;
  int nspec = 0;
  int *ctr = nullptr;  // device ints: step, status, step shadow, frame base, kernel frame base
  float *d_stf = nullptr;
  size_t nq = 0;
  // tile-local point of every Stacey and source entry, kept to regroup the
  // boundary terms when coupling entries are added
  std::vector<int> h_st_local, h_src_local;

  // With both tile groups present, the CPML tiles run on a side stream beside
  // the other tiles (the two write disjoint points and slots), joined before
  // the shared-point kernel: their longer latency hides behind the bulk.
  cudaStream_t side = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  int make_side_stream() {
    if (side || !(pml_tile0 > 0 && pml_tile0 < T.ntiles)) return SF2D_OK;
    SF2D_CUDA(cudaStreamCreateWithPriority(&side, cudaStreamNonBlocking, priority));
    SF2D_CUDA(cudaEventCreateWithFlags(&ev_fork, cudaEventDisableTiming));
    SF2D_CUDA(cudaEventCreateWithFlags(&ev_join, cudaEventDisableTiming));
    return SF2D_OK;
  }
  // parameters of the CPML tiles' kernel: its shared-memory layout is sized
  // by the layer's largest tile
  sf2d::Params pml_params() const {
    sf2d::Params Q = P;
    Q.max_q = pml_max_q;
    Q.max_local = pml_max_local;
    return Q;
  }
  template <typename F, typename... A>
  void launch_pdl(F fn, int grid, int block, size_t smem_bytes, A... args) {
    sf2d::launch_pdl(stream, launch_error, fn, grid, block, smem_bytes, args...);
  }
  cudaError_t launch_error = cudaSuccess;
  // Tiles [first, ntiles): the plain ones on the solver stream, the CPML ones
  // beside them on the side stream when there is one.  first = late_tile0
  // leaves the early tiles to launch_early.
  // kstep: steps since the counter on the device was last advanced.
  void launch_tile(bool record_prev, int stage, int first, int kstep) {
    const int rp = record_prev ? 1 : 0;
    const int nplain = pml_tile0 - first;
    if (side) {
      cudaEventRecord(ev_fork, stream);
      cudaStreamWaitEvent(side, ev_fork, 0);
      pml_fn<<<T.ntiles - pml_tile0, pml_nt, pml_smem, side>>>(pml_params(), rp, stage, pml_tile0, kstep);
      cudaEventRecord(ev_join, side);
      if (nplain > 0) tile_fn<<<nplain, lane_nt, smem, stream>>>(P, rp, stage, first, kstep);
      cudaStreamWaitEvent(stream, ev_join, 0);
      return;
    }
    if (nplain > 0) launch_pdl(tile_fn, nplain, lane_nt, smem, P, rp, stage, first, kstep);
    if (pml_tile0 < T.ntiles)
      pml_fn<<<T.ntiles - pml_tile0, pml_nt, pml_smem, stream>>>(pml_params(), rp, stage, pml_tile0, kstep);
  }
  // the early tiles [0, late_tile0) on stream s
  void launch_early(cudaStream_t s, bool record_prev, int stage, int kstep) {
    if (late_tile0 > 0) tile_fn<<<late_tile0, lane_nt, smem, s>>>(P, record_prev ? 1 : 0, stage, 0, kstep);
  }
  // tile-kernel launches of one stage of launch_tile(first)
  int tile_launches(int first) const {
    return (pml_tile0 - first > 0) + (pml_tile0 < T.ntiles);
  }
  void launch_shared(int stage, int kstep) {
    if (P.nshared == 0) return;
    const int nb = (P.nshared + sf2d::SHARED_NT - 1) / sf2d::SHARED_NT;
    if (lddrk)
      launch_pdl(sf2d::k_elastic_shared<true, false>, nb, sf2d::SHARED_NT, 0, P, stage, kstep);
    else if (kern)
      launch_pdl(sf2d::k_elastic_shared<false, true>, nb, sf2d::SHARED_NT, 0, P, stage, kstep);
    else
      launch_pdl(sf2d::k_elastic_shared<false, false>, nb, sf2d::SHARED_NT, 0, P, stage, kstep);
  }
  // the k-th step of a chunk
  void launch_step(int k) {
    for (int st = 0; st < nstage; ++st) {
      launch_tile(k > 0 && st == 0, st, 0, k);
      launch_shared(st, k);
    }
  }
  // after n steps: their last receiver samples, the step counter
  void launch_advance(int n) { launch_pdl(sf2d::k_advance, 1, 256, 0, P, n); }
  int launch_chunk(int n) {
    for (int k = 0; k < n; ++k) launch_step(k);
    launch_advance(n);
    if (launch_error != cudaSuccess) {
      const cudaError_t e = launch_error;
      launch_error = cudaSuccess;
      return sf2d::fail(SF2D_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(e));
    }
    SF2D_CUDA(cudaGetLastError());
    return SF2D_OK;
  }
  ~sf2d_solver() {
    if (graph) cudaGraphExecDestroy(graph);
    for (void *p : allocs) cudaFree(p);
    if (ev_fork) cudaEventDestroy(ev_fork);
    if (ev_join) cudaEventDestroy(ev_join);
    if (side) cudaStreamDestroy(side);
    if (stream) cudaStreamDestroy(stream);
  }
};


namespace sf2d {
// Kernel sums of an adjoint solver to the reference's element layout on the
// device, with save_kernels_elastic's scaling (save_adjoint_kernels.f90:134-141):
// one thread per element point, so that the host only receives the arrays.
// (Gathering and scaling them on the host took as long as 100 steps of a
// 64,000-element mesh.)
struct KernelScale {
  int nspec = 0;
  float *mod = nullptr;   // [3][point]: rho, kappa, mu
  float *out = nullptr;   // [3][point]: the scaled kernels
  int *lane = nullptr;    // first row of each element
  int *point = nullptr;   // device point of each element point
  // Allocates through `alloc(void **, bytes)` and uploads; point arrays in
  // reference layout.
  template <typename Alloc>
  int prepare(const sf2d_solver *A, int nspec_, const int *ibool, const float *rho, const float *kappa,
              const float *mu, Alloc alloc);
  // Kernels to host arrays, after the work queued on A's stream.
  int fetch(const sf2d_solver *A, float dt, float *rho_kl, float *kappa_kl, float *mu_kl) const;
};
static __global__ void k_scale_kernels(KernelScale K, const float2 *kmu, const float *rho_glob, float dt) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x, n = 25 * K.nspec;
  if (p >= n) return;
  const int q = p % 25, r = K.lane[p / 25] + q / 5;
  const float2 km = kmu[(static_cast<size_t>(r >> 5) * 5 + q % 5) * 32 + (r & 31)];
  const size_t sn = static_cast<size_t>(n);
  K.out[p] = -K.mod[p] * dt * rho_glob[K.point[p]];
  K.out[sn + p] = -K.mod[sn + p] * dt * km.x;
  K.out[2 * sn + p] = -2.f * K.mod[2 * sn + p] * dt * km.y;
}
template <typename Alloc>
int KernelScale::prepare(const sf2d_solver *A, int nspec_, const int *ibool, const float *rho, const float *kappa,
                         const float *mu, Alloc alloc) {
  nspec = nspec_;
  const size_t n = static_cast<size_t>(nspec) * NGLL2;
  std::vector<int> r(nspec), pt(n);
  for (int s = 0; s < nspec; ++s) r[A->T.elem_order[s]] = A->slot_lane[s];
  for (size_t p = 0; p < n; ++p) pt[p] = A->T.glob2dev[ibool[p]];
  int rc;
  if ((rc = alloc(reinterpret_cast<void **>(&mod), 3 * n * sizeof(float))) ||
      (rc = alloc(reinterpret_cast<void **>(&out), 3 * n * sizeof(float))) ||
      (rc = alloc(reinterpret_cast<void **>(&lane), r.size() * sizeof(int))) ||
      (rc = alloc(reinterpret_cast<void **>(&point), n * sizeof(int))))
    return rc;
  SF2D_CUDA(cudaMemcpy(mod, rho, n * sizeof(float), cudaMemcpyHostToDevice));
  SF2D_CUDA(cudaMemcpy(mod + n, kappa, n * sizeof(float), cudaMemcpyHostToDevice));
  SF2D_CUDA(cudaMemcpy(mod + 2 * n, mu, n * sizeof(float), cudaMemcpyHostToDevice));
  SF2D_CUDA(cudaMemcpy(lane, r.data(), r.size() * sizeof(int), cudaMemcpyHostToDevice));
  SF2D_CUDA(cudaMemcpy(point, pt.data(), n * sizeof(int), cudaMemcpyHostToDevice));
  return SF2D_OK;
}
inline int KernelScale::fetch(const sf2d_solver *A, float dt, float *rho_kl, float *kappa_kl, float *mu_kl) const {
  const size_t n = static_cast<size_t>(nspec) * NGLL2;
  k_scale_kernels<<<static_cast<unsigned>((n + 255) / 256), 256, 0, A->stream>>>(*this, A->P.kmu_kl, A->P.rho_kl_glob, dt);
  SF2D_CUDA(cudaGetLastError());
  SF2D_CUDA(cudaMemcpyAsync(rho_kl, out, n * sizeof(float), cudaMemcpyDeviceToHost, A->stream));
  SF2D_CUDA(cudaMemcpyAsync(kappa_kl, out + n, n * sizeof(float), cudaMemcpyDeviceToHost, A->stream));
  SF2D_CUDA(cudaMemcpyAsync(mu_kl, out + 2 * n, n * sizeof(float), cudaMemcpyDeviceToHost, A->stream));
  SF2D_CUDA(cudaStreamSynchronize(A->stream));
  return SF2D_OK;
}
}  // namespace sf2d

// Builds a solver; `kern` selects the adjoint variant that accumulates
// sensitivity kernels against forward displacement frames.
// late_elem (may be NULL): per element 1 when another domain reads or writes
// one of its points (fluid-solid coupling); those elements get tiles of their
// own, launched after the other domain's step, and the rest may run beside it
int sf2d_create_solver_internal(const sf2d_elastic_desc *d, bool kern, sf2d_solver **out, const uint8_t *late_elem);

// Zeroes every wavefield, memory variable, kernel sum and counter of a solver.
int sf2d_reset_solver(sf2d_solver *S);

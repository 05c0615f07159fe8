// Gaussian smoothing of sensitivity kernels (the post-gradient step of an
// inversion): the computation of src/tomography/postprocess_sensitivity_kernels/
// smooth_sem.F90:63-467 (CPU) and of src/gpu/kernels/process_smooth.cu:37-116.
//
// Every element GLL point i gets
//   out_k(i) = sum_j G(i,j) J_j w_j f_k(j) / sum_j G(i,j) J_j w_j,
//   G = exp(-(x_i - x_j)^2 / (2 sigma_h^2) - (z_i - z_j)^2 / (2 sigma_v^2)),
// the sums running over every element GLL point j (w_j = wxgll * wzgll of
// its position, J_j its Jacobian).  The reference's CPU program sums over all
// pairs; this kernel sums over the points within `cutoff` standard
// deviations (an ellipse), so the weight left out is below exp(-cutoff^2/2)
// of the nearest one.
//
// Coordinates are scaled (x / sigma_h, z / sigma_v).  The host sorts the
// elements, not the points, into cells of about one standard deviation; a CTA
// takes the targets of up to SM_TE elements of one cell, walks the cells
// around them, keeps the elements whose bounding box comes within the cutoff
// of its own box (in order: the result does not depend on the schedule) and
// stages their points in shared memory.  What bounds it is the arithmetic of
// a pair: one expf, one conversion and 1 + nfields double multiply-adds; the
// products J w f are formed in double when they are staged, exactly, so that a
// pair needs no further conversion, and two targets per thread share each
// staged point.  Walking cells of the cutoff's size point by point visited
// three times the pairs that count and converted three operands for each: a
// 200 x 80 element mesh (400,000 points, three fields, sigma of a few elements)
// took 54.0 ms that way, and takes 24.9 ms (host sorting and copies included).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "sf2d_b200.h"
#include "sf2d_runtime.h"

namespace {

constexpr int SM_NT = 128;  // threads of a CTA, two targets each
constexpr int SM_TE = 10;   // target elements of a CTA: 250 of its 256 places
constexpr int SM_SE = 10;   // source elements staged at a time

struct SmoothArgs {
  const float *x, *z, *jac;   // element GLL points
  const float *val;           // [field][point]
  const int *elem;            // sorted elements
  const float4 *box;          // their bounding boxes: xmin, xmax, zmin, zmax, scaled
  const int *cell_start;      // ncx * ncz + 1 offsets into the sorted elements
  const int2 *blocks;         // per CTA: its range of sorted elements
  float *out;                 // [field][point]
  size_t npoint;
  int ncx, ncz;
  float x0, z0, cellx, cellz, halfx, halfz;  // cell grid of the element centres; largest half extents
  float sigma_h, sigma_v, cutoff, cut2;
  float w[25];
};

template <int NF>
__global__ void __launch_bounds__(SM_NT) k_smooth(const SmoothArgs A) {
  __shared__ float2 s_pos[SM_SE * 25];
  __shared__ double s_w[SM_SE * 25], s_wv[NF][SM_SE * 25];
  __shared__ int s_list[SM_NT], s_cnt[SM_NT / 32 + 1];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int2 blk = A.blocks[blockIdx.x];
  const int ntarget = (blk.y - blk.x) * 25;
  float2 t[2];
  size_t tp[2];
  double norm[2] = {0.0, 0.0}, acc[2][NF] = {};
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int k = min(tid + r * SM_NT, ntarget - 1);
    tp[r] = static_cast<size_t>(A.elem[blk.x + k / 25]) * 25 + k % 25;
    t[r] = make_float2(A.x[tp[r]] / A.sigma_h, A.z[tp[r]] / A.sigma_v);
  }
  float4 b = A.box[blk.x];
  for (int k = blk.x + 1; k < blk.y; ++k) {
    const float4 o = A.box[k];
    b = make_float4(fminf(b.x, o.x), fmaxf(b.y, o.y), fminf(b.z, o.z), fmaxf(b.w, o.w));
  }
  // cells whose elements can come within the cutoff, one more on each side for rounding
  auto cell = [](float v, float v0, float size, int n) {
    return static_cast<int>(fminf(fmaxf(floorf((v - v0) / size), 0.f), static_cast<float>(n - 1)));
  };
  const float rx = A.cutoff + A.halfx, rz = A.cutoff + A.halfz;
  const int cx0 = max(0, cell(b.x - rx, A.x0, A.cellx, A.ncx) - 1), cx1 = min(A.ncx - 1, cell(b.y + rx, A.x0, A.cellx, A.ncx) + 1);
  const int cz0 = max(0, cell(b.z - rz, A.z0, A.cellz, A.ncz) - 1), cz1 = min(A.ncz - 1, cell(b.w + rz, A.z0, A.cellz, A.ncz) + 1);
  const float reach2 = A.cut2 * 1.0001f;
  for (int c = cz0; c <= cz1; ++c) {
    const int e0 = A.cell_start[static_cast<size_t>(c) * A.ncx + cx0], e1 = A.cell_start[static_cast<size_t>(c) * A.ncx + cx1 + 1];
    for (int base = e0; base < e1; base += SM_NT) {
      // the batch's elements within reach, in order
      bool hit = false;
      if (base + tid < e1) {
        const float4 o = A.box[base + tid];
        const float dx = fmaxf(0.f, fmaxf(o.x - b.y, b.x - o.y)), dz = fmaxf(0.f, fmaxf(o.z - b.w, b.z - o.w));
        hit = dx * dx + dz * dz <= reach2;
      }
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      __syncthreads();  // the previous batch's list and points are done with
      if (lane == 0) s_cnt[warp] = __popc(m);
      __syncthreads();
      int before = 0, total = 0;
#pragma unroll
      for (int k = 0; k < SM_NT / 32; ++k) {
        before += k < warp ? s_cnt[k] : 0;
        total += s_cnt[k];
      }
      if (hit) s_list[before + __popc(m & ((1u << lane) - 1u))] = A.elem[base + tid];
      for (int l0 = 0; l0 < total; l0 += SM_SE) {
        const int np = min(SM_SE, total - l0) * 25;
        __syncthreads();
        for (int k = tid; k < np; k += SM_NT) {
          const size_t p = static_cast<size_t>(s_list[l0 + k / 25]) * 25 + k % 25;
          s_pos[k] = make_float2(A.x[p] / A.sigma_h, A.z[p] / A.sigma_v);
          const double wj = static_cast<double>(A.jac[p] * A.w[k % 25]);
          s_w[k] = wj;
#pragma unroll
          for (int f = 0; f < NF; ++f) s_wv[f][k] = wj * static_cast<double>(A.val[f * A.npoint + p]);
        }
        __syncthreads();
#pragma unroll 2
        for (int k = 0; k < np; ++k) {
          const float2 q = s_pos[k];
          const double wj = s_w[k];
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const float ddx = t[r].x - q.x, ddz = t[r].y - q.y;
            const float r2 = ddx * ddx + ddz * ddz;
            if (r2 <= A.cut2) {  // what lies beyond adds nothing, whatever its value
              const double g = static_cast<double>(expf(-0.5f * r2));
              norm[r] += g * wj;
#pragma unroll
              for (int f = 0; f < NF; ++f) acc[r][f] += g * s_wv[f][k];
            }
          }
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 2; ++r)
    if (tid + r * SM_NT < ntarget)
#pragma unroll
      for (int f = 0; f < NF; ++f) A.out[f * A.npoint + tp[r]] = static_cast<float>(acc[r][f] / norm[r]);
}

}  // namespace

extern "C" int sf2d_smooth(int nspec, const float *x, const float *z, const float *jacobian, const float *wgll_sq,
                           int nfields, const float *fields, float sigma_h, float sigma_v, float cutoff, float *out,
                           void *stream_v) {
  if (nspec < 1 || !x || !z || !jacobian || !wgll_sq || !fields || !out)
    return fail(SF2D_ERR_INVALID, "sf2d_smooth: null argument");
  if (nfields < 1 || nfields > SF2D_SMOOTH_MAX_FIELDS)
    return fail(SF2D_ERR_INVALID, "sf2d_smooth: 1 to SF2D_SMOOTH_MAX_FIELDS fields per call");
  if (!(sigma_h > 0.f) || !(sigma_v > 0.f) || !(cutoff > 0.f))
    return fail(SF2D_ERR_INVALID, "sf2d_smooth: sigma_h, sigma_v and cutoff must be positive");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  const size_t n = static_cast<size_t>(nspec) * 25;
  if (n > static_cast<size_t>(INT32_MAX)) return fail(SF2D_ERR_INVALID, "sf2d_smooth: too many points");
  // bounding boxes and centres of the elements in scaled coordinates
  const size_t ne = static_cast<size_t>(nspec);
  std::vector<float4> box(ne);
  std::vector<float2> mid(ne);
  float xmin = INFINITY, xmax = -INFINITY, zmin = INFINITY, zmax = -INFINITY;
  SmoothArgs A{};
  for (size_t k = 0; k < ne; ++k) {
    float4 b = make_float4(INFINITY, -INFINITY, INFINITY, -INFINITY);
    for (size_t p = 25 * k; p < 25 * k + 25; ++p) {
      const float sx = x[p] / sigma_h, sz = z[p] / sigma_v;
      b = make_float4(std::min(b.x, sx), std::max(b.y, sx), std::min(b.z, sz), std::max(b.w, sz));
    }
    box[k] = b;
    mid[k] = make_float2(0.5f * (b.x + b.y), 0.5f * (b.z + b.w));
    xmin = std::min(xmin, b.x);
    xmax = std::max(xmax, b.y);
    zmin = std::min(zmin, b.z);
    zmax = std::max(zmax, b.w);
    A.halfx = std::max(A.halfx, 0.5f * (b.y - b.x) * 1.001f);
    A.halfz = std::max(A.halfz, 0.5f * (b.w - b.z) * 1.001f);
  }
  const long long kx = std::max(1LL, static_cast<long long>((xmax - xmin) / cutoff) + 1);
  const long long kz = std::max(1LL, static_cast<long long>((zmax - zmin) / cutoff) + 1);
  if (kx * kz > (1LL << 28)) return fail(SF2D_ERR_INVALID, "sf2d_smooth: sigma too small for the mesh extent");
  // cells of one standard deviation or three mean elements, larger when the
  // mesh fills little of its extent
  double sumx = 0.0, sumz = 0.0;
  for (size_t k = 0; k < ne; ++k) {
    sumx += box[k].y - box[k].x;
    sumz += box[k].w - box[k].z;
  }
  A.cellx = std::max(1.f, static_cast<float>(3.0 * sumx / ne));
  A.cellz = std::max(1.f, static_cast<float>(3.0 * sumz / ne));
  auto count = [](float lo, float hi, float size) { return std::max(1LL, static_cast<long long>((hi - lo) / size) + 1); };
  while (static_cast<double>(count(xmin, xmax, A.cellx)) * static_cast<double>(count(zmin, zmax, A.cellz)) >
         4.0 * ne + 1024.0) {
    A.cellx *= 1.5f;
    A.cellz *= 1.5f;
  }
  const long long ncx = count(xmin, xmax, A.cellx), ncz = count(zmin, zmax, A.cellz);
  std::vector<int> cell_of(ne), start(static_cast<size_t>(ncx * ncz) + 1, 0);
  for (size_t k = 0; k < ne; ++k) {
    const long long cx = std::min<long long>(ncx - 1, std::max<long long>(0, static_cast<long long>((mid[k].x - xmin) / A.cellx)));
    const long long cz = std::min<long long>(ncz - 1, std::max<long long>(0, static_cast<long long>((mid[k].y - zmin) / A.cellz)));
    cell_of[k] = static_cast<int>(cz * ncx + cx);
    ++start[cell_of[k] + 1];
  }
  for (size_t c = 0; c + 1 < start.size(); ++c) start[c + 1] += start[c];
  std::vector<int> fill(start.begin(), start.end() - 1), elem(ne);
  std::vector<float4> sbox(ne);
  for (size_t k = 0; k < ne; ++k) {
    const int o = fill[cell_of[k]]++;
    elem[o] = static_cast<int>(k);
    sbox[o] = box[k];
  }
  std::vector<int2> blocks;
  for (size_t c = 0; c + 1 < start.size(); ++c) {
    const int m = start[c + 1] - start[c], nb = (m + SM_TE - 1) / SM_TE;
    for (int k = 0; k < nb; ++k)  // even shares
      blocks.push_back(make_int2(start[c] + static_cast<int>(static_cast<long long>(m) * k / nb),
                                 start[c] + static_cast<int>(static_cast<long long>(m) * (k + 1) / nb)));
  }
  // device buffers, one allocation
  size_t bytes = 0;
  auto take = [&](size_t want) {
    const size_t at = bytes;
    bytes += (want + 255) / 256 * 256;
    return at;
  };
  const size_t fb = n * sizeof(float);
  const size_t o_x = take(fb), o_z = take(fb), o_jac = take(fb), o_val = take(fb * nfields), o_out = take(fb * nfields);
  const size_t o_elem = take(ne * sizeof(int)), o_box = take(ne * sizeof(float4));
  const size_t o_start = take(start.size() * sizeof(int)), o_blk = take(blocks.size() * sizeof(int2));
  char *buf = nullptr;
  cudaError_t e = cudaMalloc(&buf, bytes);
  if (e != cudaSuccess)
    return fail(e == cudaErrorMemoryAllocation ? SF2D_ERR_OOM : SF2D_ERR_CUDA, "sf2d_smooth: cudaMalloc");
  struct Free {
    char *p;
    ~Free() { cudaFree(p); }
  } guard{buf};
  auto up = [&](size_t at, const void *src, size_t size) {
    return cudaMemcpyAsync(buf + at, src, size, cudaMemcpyHostToDevice, stream);
  };
  SF2D_CUDA(up(o_x, x, fb));
  SF2D_CUDA(up(o_z, z, fb));
  SF2D_CUDA(up(o_jac, jacobian, fb));
  SF2D_CUDA(up(o_val, fields, fb * nfields));
  SF2D_CUDA(up(o_elem, elem.data(), ne * sizeof(int)));
  SF2D_CUDA(up(o_box, sbox.data(), ne * sizeof(float4)));
  SF2D_CUDA(up(o_start, start.data(), start.size() * sizeof(int)));
  SF2D_CUDA(up(o_blk, blocks.data(), blocks.size() * sizeof(int2)));
  A.x = reinterpret_cast<float *>(buf + o_x);
  A.z = reinterpret_cast<float *>(buf + o_z);
  A.jac = reinterpret_cast<float *>(buf + o_jac);
  A.val = reinterpret_cast<float *>(buf + o_val);
  A.out = reinterpret_cast<float *>(buf + o_out);
  A.elem = reinterpret_cast<int *>(buf + o_elem);
  A.box = reinterpret_cast<float4 *>(buf + o_box);
  A.cell_start = reinterpret_cast<int *>(buf + o_start);
  A.blocks = reinterpret_cast<int2 *>(buf + o_blk);
  A.npoint = n;
  A.ncx = static_cast<int>(ncx);
  A.ncz = static_cast<int>(ncz);
  A.x0 = xmin;
  A.z0 = zmin;
  A.sigma_h = sigma_h;
  A.sigma_v = sigma_v;
  A.cutoff = cutoff;
  A.cut2 = cutoff * cutoff;
  for (int q = 0; q < 25; ++q) A.w[q] = wgll_sq[q];
  void (*const fn[SF2D_SMOOTH_MAX_FIELDS])(SmoothArgs) = {k_smooth<1>, k_smooth<2>, k_smooth<3>, k_smooth<4>};
  fn[nfields - 1]<<<static_cast<unsigned>(blocks.size()), SM_NT, 0, stream>>>(A);
  SF2D_CUDA(cudaGetLastError());
  SF2D_CUDA(cudaMemcpyAsync(out, A.out, fb * nfields, cudaMemcpyDeviceToHost, stream));
  SF2D_CUDA(cudaStreamSynchronize(stream));
  return SF2D_OK;
}

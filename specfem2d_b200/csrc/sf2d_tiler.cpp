// Host-side tiler (see sf2d_tiler.h).
#include "sf2d_tiler.h"

#include <algorithm>
#include <cmath>
#include <numeric>
#include <unordered_map>

namespace sf2d {

namespace {

// Connected part of every element (elements that share a corner point), parts
// numbered by their first element.
std::vector<int> mesh_parts(int nspec, int nglob, const int *ibool) {
  std::vector<int> root(nspec), owner(nglob, -1);
  std::iota(root.begin(), root.end(), 0);
  auto find = [&](int e) {
    while (root[e] != e) e = root[e] = root[root[e]];
    return e;
  };
  constexpr int corner[4] = {0, NGLL - 1, NGLL2 - NGLL, NGLL2 - 1};
  for (int e = 0; e < nspec; ++e)
    for (int q : corner) {
      int &o = owner[ibool[static_cast<size_t>(e) * NGLL2 + q]];
      if (o < 0) {
        o = e;
        continue;
      }
      const int a = find(e), b = find(o);
      if (a != b) root[std::max(a, b)] = std::min(a, b);
    }
  for (int e = 0; e < nspec; ++e) root[e] = find(e);
  return root;
}

// Cuts order[b, e) into pieces of `te` elements (the last one the rest) by
// recursive bisection across the longer side of the bounding box.  key: two
// integer coordinates per element in units well below an element, so that
// rounding noise between the elements of one mesh column does not fray a cut.
struct Bisection {
  const std::vector<int> &key;
  std::vector<int> &order;
  int te;
  std::vector<std::pair<int, int>> &pieces;
  void cut(int b, int e) {
    const int nt = (e - b + te - 1) / te;
    if (nt <= 1) {
      pieces.emplace_back(b, e);
      return;
    }
    int lo[2] = {INT32_MAX, INT32_MAX}, hi[2] = {INT32_MIN, INT32_MIN};
    for (int k = b; k < e; ++k)
      for (int c = 0; c < 2; ++c) {
        const int v = key[2 * order[k] + c];
        lo[c] = std::min(lo[c], v);
        hi[c] = std::max(hi[c], v);
      }
    const int ax = hi[0] - lo[0] >= hi[1] - lo[1] ? 0 : 1;
    const int mid = b + te * (nt / 2);
    std::nth_element(order.begin() + b, order.begin() + mid, order.begin() + e, [&](int p, int q) {
      const int vp = key[2 * p + ax], vq = key[2 * q + ax];
      if (vp != vq) return vp < vq;
      const int wp = key[2 * p + 1 - ax], wq = key[2 * q + 1 - ax];
      return wp != wq ? wp < wq : p < q;
    });
    cut(b, mid);
    cut(mid, e);
  }
};

}  // namespace

int Tiling::local_id(int tile, int glob) const {
  const TileInfo &t = tiles[tile];
  const int dev = glob2dev[glob];
  if (dev >= t.int_begin && dev < t.int_begin + t.n_int) return dev - t.int_begin;
  for (int k = 0; k < t.n_sh; ++k)
    if (sh_ids[t.sh_off + k] == dev) return t.n_int + k;
  return -1;
}

std::string build_tiling(int nspec, int nglob, const int *ibool, const double *centroid_xz,
                         int tile_elems, Tiling &T, const int *elem_group, int ngroups,
                         const int *group_tile_elems, int nlaned) {
  if (nspec <= 0 || nglob <= 0 || !ibool) return "empty mesh";
  if (tile_elems < 1 || tile_elems > 256) return "tile_elems must be in [1, 256]";
  if (ngroups < 1 || ngroups > 8) return "ngroups must be in [1, 8]";
  if (group_tile_elems)
    for (int k = 0; k < ngroups; ++k)
      if (group_tile_elems[k] < 1 || group_tile_elems[k] > 256) return "tile_elems must be in [1, 256]";
  for (long long k = 0; k < static_cast<long long>(nspec) * NGLL2; ++k)
    if (ibool[k] < 0 || ibool[k] >= nglob) return "ibool entry out of range";
  if (elem_group)
    for (int e = 0; e < nspec; ++e)
      if (elem_group[e] < 0 || elem_group[e] >= ngroups) return "element group out of range";
  auto group = [&](int e) { return elem_group ? elem_group[e] : 0; };

  // 1. elements by group and connected part, each cut into tiles; elements
  //    ascending inside a tile
  T = Tiling();
  std::vector<int> order(nspec);
  std::iota(order.begin(), order.end(), 0);
  std::vector<std::pair<int, int>> pieces;
  std::vector<int> part;
  if (centroid_xz) {
    part = mesh_parts(nspec, nglob, ibool);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
      return group(a) != group(b) ? group(a) < group(b) : part[a] < part[b];
    });
  } else if (elem_group) {
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return group(a) < group(b); });
  }
  T.group_tile_begin.assign(ngroups + 1, 0);
  std::vector<int> key;
  if (centroid_xz) key.resize(2 * static_cast<size_t>(nspec));
  for (int b = 0; b < nspec;) {
    const int g = group(order[b]);
    const int te = group_tile_elems ? group_tile_elems[g] : tile_elems;
    int e = b + 1;
    if (centroid_xz) {
      while (e < nspec && group(order[e]) == g && part[order[e]] == part[order[b]]) ++e;
      double lo[2] = {1e300, 1e300}, hi[2] = {-1e300, -1e300};
      for (int k = b; k < e; ++k)
        for (int c = 0; c < 2; ++c) {
          lo[c] = std::min(lo[c], centroid_xz[2 * static_cast<size_t>(order[k]) + c]);
          hi[c] = std::max(hi[c], centroid_xz[2 * static_cast<size_t>(order[k]) + c]);
        }
      // a unit of about 1/8 of an element, and at most 2^30 units
      const double ext = std::max(hi[0] - lo[0], hi[1] - lo[1]);
      double unit = std::sqrt(std::max((hi[0] - lo[0]) * (hi[1] - lo[1]), 1e-6 * ext * ext) / (e - b)) / 7.3;
      unit = std::max(unit, std::max(ext, 1e-30) / 1e9);
      for (int k = b; k < e; ++k)
        for (int c = 0; c < 2; ++c) {
          const size_t p = 2 * static_cast<size_t>(order[k]) + c;
          key[p] = static_cast<int>((centroid_xz[p] - lo[c]) / unit + 0.3);
        }
      Bisection{key, order, te, pieces}.cut(b, e);
    } else {
      while (e < nspec && e - b < te && group(order[e]) == g) ++e;
      pieces.emplace_back(b, e);
    }
    T.group_tile_begin[g + 1] = static_cast<int>(pieces.size());
    b = e;
  }
  for (int k = 1; k <= ngroups; ++k) T.group_tile_begin[k] = std::max(T.group_tile_begin[k], T.group_tile_begin[k - 1]);
  for (const auto &pc : pieces) std::sort(order.begin() + pc.first, order.begin() + pc.second);
  const int ntiles = static_cast<int>(pieces.size());
  T.ntiles = ntiles;
  T.nglob = nglob;
  T.nelem = nspec;
  T.tiles.assign(ntiles, TileInfo{});
  T.elem_tile.assign(nspec, -1);
  for (int t = 0; t < ntiles; ++t)
    for (int k = pieces[t].first; k < pieces[t].second; ++k) T.elem_tile[order[k]] = t;
  const int ntiles_laned = T.group_tile_begin[std::min(nlaned, ngroups)];

  // 2. how many tiles touch each point
  std::vector<int> last(nglob, -1), touch(nglob, 0);
  for (int t = 0; t < ntiles; ++t)
    for (int k = pieces[t].first; k < pieces[t].second; ++k)
      for (int q = 0; q < NGLL2; ++q) {
        const int g = ibool[static_cast<size_t>(order[k]) * NGLL2 + q];
        if (last[g] != t) {
          last[g] = t;
          ++touch[g];
        }
      }
  for (int g = 0; g < nglob; ++g)
    if (touch[g] == 0) return "a global point is not referenced by any element";

  // 3. segments: the shared points by the set of tiles that touch them,
  //    numbered as the tiles (in order) first meet them
  std::vector<int> sidx(nglob, -1);  // global -> shared index
  int nsh = 0;
  for (int g = 0; g < nglob; ++g)
    if (touch[g] > 1) sidx[g] = nsh++;
  std::vector<int> toff(nsh + 1, 0), tlist, seg_of(nsh, -1), pos(nsh, 0);
  for (int g = 0; g < nglob; ++g)
    if (sidx[g] >= 0) toff[sidx[g] + 1] = touch[g];
  for (int k = 0; k < nsh; ++k) toff[k + 1] += toff[k];
  tlist.resize(toff[nsh]);
  {
    std::vector<int> fill(toff.begin(), toff.end() - 1);
    std::fill(last.begin(), last.end(), -1);
    for (int t = 0; t < ntiles; ++t)
      for (int k = pieces[t].first; k < pieces[t].second; ++k)
        for (int q = 0; q < NGLL2; ++q) {
          const int g = ibool[static_cast<size_t>(order[k]) * NGLL2 + q];
          if (sidx[g] < 0 || last[g] == t) continue;
          last[g] = t;
          tlist[fill[sidx[g]]++] = t;
        }
  }
  std::vector<int> seg_first, seg_count;  // a point of the segment (its tile list), its points
  {
    std::unordered_multimap<uint64_t, int> seen;
    auto same = [&](int a, int b) {
      return toff[a + 1] - toff[a] == toff[b + 1] - toff[b] &&
             std::equal(tlist.begin() + toff[a], tlist.begin() + toff[a + 1], tlist.begin() + toff[b]);
    };
    int prev = -1;
    auto find = [&](int k) {
      if (prev >= 0 && same(k, seg_first[prev])) return prev;
      uint64_t h = 1469598103934665603ull;
      for (int x = toff[k]; x < toff[k + 1]; ++x) h = (h ^ static_cast<uint64_t>(tlist[x])) * 1099511628211ull;
      const auto r = seen.equal_range(h);
      for (auto it = r.first; it != r.second; ++it)
        if (same(k, seg_first[it->second])) return it->second;
      seg_first.push_back(k);
      seg_count.push_back(0);
      const int s = static_cast<int>(seg_first.size()) - 1;
      seen.emplace(h, s);
      return s;
    };
    for (int t = 0; t < ntiles; ++t) {
      const int b = pieces[t].first, ne = pieces[t].second - b;
      for (int q = 0; q < NGLL2; ++q)
        for (int k = 0; k < ne; ++k) {
          const int x = sidx[ibool[static_cast<size_t>(order[b + k]) * NGLL2 + q]];
          if (x < 0 || seg_of[x] >= 0) continue;
          prev = find(x);
          seg_of[x] = prev;
          pos[x] = seg_count[prev]++;
        }
    }
  }
  const int nsegs = static_cast<int>(seg_first.size());
  T.nshared = nsh;
  T.shared_begin = nglob - nsh;
  T.shp_off.assign(nsh + 1, 0);
  std::vector<int> seg_dev(nsegs), seg_slot(nsegs), seg_rank(nsegs, 0), seg_tile(nsegs, -1), seg_local(nsegs, 0);
  {
    int dev = T.shared_begin, slot = 0;
    for (int s = 0; s < nsegs; ++s) {
      seg_dev[s] = dev;
      seg_slot[s] = slot;
      for (int i = 0; i < seg_count[s]; ++i) {
        slot += toff[seg_first[s] + 1] - toff[seg_first[s]];
        T.shp_off[dev + i + 1 - T.shared_begin] = slot;
      }
      dev += seg_count[s];
    }
  }

  // 4. device numbering, local ids, colours or phases, local ibool
  T.glob2dev.assign(nglob, -1);
  T.dev2glob.assign(nglob, -1);
  T.elem_order.reserve(nspec);
  T.lib.reserve(static_cast<size_t>(nspec) * NGLL2 + 8 * static_cast<size_t>(ntiles));
  std::vector<int> local(nglob, -1);       // local id of an interior point in the tile at hand
  std::fill(last.begin(), last.end(), -1);  // tile that set it
  std::vector<int> lid, cls, idx, my;
  std::vector<uint32_t> used;
  std::vector<uint64_t> busy;  // 128 phase bits per local point
  int next_dev = 0;
  for (int g = 0; g < nglob; ++g)
    if (sidx[g] >= 0) {
      T.glob2dev[g] = seg_dev[seg_of[sidx[g]]] + pos[sidx[g]];
      T.dev2glob[T.glob2dev[g]] = g;
    }
  for (int t = 0; t < ntiles; ++t) {
    TileInfo &ti = T.tiles[t];
    const int b = pieces[t].first, ne = pieces[t].second - b;
    const bool laned = t < ntiles_laned;
    ti.int_begin = next_dev;
    my.clear();
    auto visit = [&](int k, int q) {
      const int g = ibool[static_cast<size_t>(order[b + k]) * NGLL2 + q];
      if (last[g] == t) return;
      last[g] = t;
      if (sidx[g] < 0) {
        local[g] = next_dev - ti.int_begin;
        T.glob2dev[g] = next_dev;
        T.dev2glob[next_dev++] = g;
      } else {
        const int s = seg_of[sidx[g]];
        if (seg_tile[s] != t) {
          seg_tile[s] = t;
          my.push_back(s);
        }
      }
    };
    if (laned)
      for (int i = 0; i < NGLL; ++i)
        for (int k = 0; k < ne; ++k)
          for (int j = 0; j < NGLL; ++j) visit(k, NGLL * j + i);
    else
      for (int k = 0; k < ne; ++k)
        for (int q = 0; q < NGLL2; ++q) visit(k, q);
    ti.n_int = next_dev - ti.int_begin;
    ti.sh_off = static_cast<int>(T.sh_ids.size());
    std::sort(my.begin(), my.end());
    int nl = ti.n_int;
    for (int s : my) {
      const int nt = toff[seg_first[s] + 1] - toff[seg_first[s]];
      seg_local[s] = nl;
      for (int i = 0; i < seg_count[s]; ++i) {
        T.sh_ids.push_back(seg_dev[s] + i);
        T.sh_slot.push_back(seg_slot[s] + i * nt + seg_rank[s]);
      }
      ++seg_rank[s];
      nl += seg_count[s];
    }
    ti.n_sh = nl - ti.n_int;
    if (nl > 8191) return "too many local points in a tile";
    T.max_local = std::max(T.max_local, nl);
    T.max_elems = std::max(T.max_elems, ne);
    lid.resize(static_cast<size_t>(ne) * NGLL2);
    for (int k = 0; k < ne; ++k)
      for (int q = 0; q < NGLL2; ++q) {
        const int g = ibool[static_cast<size_t>(order[b + k]) * NGLL2 + q];
        lid[static_cast<size_t>(k) * NGLL2 + q] = sidx[g] < 0 ? local[g] : seg_local[seg_of[sidx[g]]] + pos[sidx[g]];
      }
    ti.elem_base = static_cast<int>(T.elem_order.size());
    ti.nelem = ne;
    ti.ncol = 0;
    for (int c = 0; c < MAX_COLOURS; ++c) ti.col_end[c] = 0;
    idx.resize(ne);
    std::iota(idx.begin(), idx.end(), 0);
    T.phases.resize(T.elem_order.size() + ne, 0u);
    if (laned) {
      ti.lane0 = T.nlanes;
      T.nlanes += (5 * ne + 31) / 32 * 32;
      busy.assign(2 * static_cast<size_t>(nl), 0);
      for (int c = 0; c < PHASE_CLASSES; ++c)
        for (int k = 0; k < ne; ++k) {
          uint64_t m[2] = {0, 0};
          for (int q = 0; q < NGLL2; ++q)
            if (phase_class(q) == c) {
              const size_t l = lid[static_cast<size_t>(k) * NGLL2 + q];
              m[0] |= busy[2 * l];
              m[1] |= busy[2 * l + 1];
            }
          int p = c;
          while (p < MAX_PHASES && (m[p >> 6] >> (p & 63)) & 1u) ++p;
          if (p == MAX_PHASES) return "a point is held by too many elements of a tile";
          for (int q = 0; q < NGLL2; ++q)
            if (phase_class(q) == c) busy[2 * static_cast<size_t>(lid[static_cast<size_t>(k) * NGLL2 + q]) + (p >> 6)] |= 1ull << (p & 63);
          T.phases[ti.elem_base + k] |= static_cast<uint32_t>(p) << (8 * c);
          ti.ncol = std::max(ti.ncol, p + 1);
        }
    } else {
      auto colour = [&](const std::vector<int> &seq) {
        used.assign(nl, 0u);
        cls.assign(ne, 0);
        for (int k : seq) {
          uint32_t m = 0;
          for (int q = 0; q < NGLL2; ++q) m |= used[lid[static_cast<size_t>(k) * NGLL2 + q]];
          int c = 0;
          while (c < MAX_COLOURS && (m >> c) & 1u) ++c;
          if (c == MAX_COLOURS) return false;
          cls[k] = c;
          for (int q = 0; q < NGLL2; ++q) used[lid[static_cast<size_t>(k) * NGLL2 + q]] |= 1u << c;
        }
        return true;
      };
      if (!colour(idx)) {
        // elements numbered at random can use up the colours; along the tile's
        // rows a structured mesh takes four or five whatever its numbering
        if (centroid_xz)
          std::sort(idx.begin(), idx.end(), [&](int a, int c) {
            const size_t p = 2 * static_cast<size_t>(order[b + a]), r = 2 * static_cast<size_t>(order[b + c]);
            if (key[p + 1] != key[r + 1]) return key[p + 1] < key[r + 1];
            return key[p] != key[r] ? key[p] < key[r] : a < c;
          });
        if (!centroid_xz || !colour(idx)) return "element colouring needs more than 8 colours in a tile";
        std::iota(idx.begin(), idx.end(), 0);
      }
      std::stable_sort(idx.begin(), idx.end(), [&](int a, int c) { return cls[a] < cls[c]; });
    }
    while (T.lib.size() % 8) T.lib.push_back(0);
    ti.lib_off = static_cast<int>(T.lib.size());
    for (int s = 0; s < ne; ++s) {
      const int k = idx[s];
      T.elem_order.push_back(order[b + k]);
      for (int q = 0; q < NGLL2; ++q) T.lib.push_back(static_cast<uint16_t>(lid[static_cast<size_t>(k) * NGLL2 + q]));
      if (!laned) {
        ti.col_end[cls[k]] = s + 1;
        ti.ncol = std::max(ti.ncol, cls[k] + 1);
      }
    }
    if (!laned)
      for (int c = 1; c < ti.ncol; ++c) ti.col_end[c] = std::max(ti.col_end[c], ti.col_end[c - 1]);
  }
  // the kernel copies each coloured tile's local ibool in 16-byte chunks
  while (T.lib.size() % 8) T.lib.push_back(0);
  return "";
}

}  // namespace sf2d

// Host-only diagnostic (declared in include/sf2d_b200.h): builds a tiling and
// checks its invariants without touching the GPU.
extern "C" int sf2d_tiling_stats(int nspec, int nglob, const int *ibool, const double *centroid_xz,
                                 int tile_elems, long long *out8) {
  using namespace sf2d;
  if (!out8) return -1;
  Tiling T;
  const std::string err = build_tiling(nspec, nglob, ibool, centroid_xz, tile_elems, T);
  if (!err.empty()) return -1;
  // every global point has exactly one device id
  std::vector<int> seen(nglob, 0);
  for (int d = 0; d < nglob; ++d) {
    const int g = T.dev2glob[d];
    if (g < 0 || g >= nglob || T.glob2dev[g] != d) return -2;
    ++seen[g];
  }
  for (int g = 0; g < nglob; ++g)
    if (seen[g] != 1) return -2;
  long long max_col = 0, nint = 0;
  for (int t = 0; t < T.ntiles; ++t) {
    const TileInfo &ti = T.tiles[t];
    nint += ti.n_int;
    max_col = std::max<long long>(max_col, ti.ncol);
    // local ibool maps back to the original ibool
    for (int s = ti.elem_base; s < ti.elem_base + ti.nelem; ++s) {
      const int e = T.elem_order[s];
      for (int q = 0; q < NGLL2; ++q) {
        const int l = T.lib[static_cast<size_t>(ti.lib_off) + static_cast<size_t>(s - ti.elem_base) * NGLL2 + q];
        const int g = ibool[static_cast<size_t>(e) * NGLL2 + q];
        const int dev = l < ti.n_int ? ti.int_begin + l : T.sh_ids[ti.sh_off + l - ti.n_int];
        if (T.dev2glob[dev] != g) return -3;
      }
    }
    // no two elements of one colour share a local point
    int cb = 0;
    for (int c = 0; c < ti.ncol; ++c) {
      std::vector<char> mark(ti.n_int + ti.n_sh, 0);
      for (int s = cb; s < ti.col_end[c]; ++s)
        for (int q = 0; q < NGLL2; ++q) {
          const int l = T.lib[static_cast<size_t>(ti.lib_off) + static_cast<size_t>(s) * NGLL2 + q];
          if (mark[l]) return -4;
          mark[l] = 1;
        }
      cb = ti.col_end[c];
    }
    if (cb != ti.nelem) return -5;
  }
  // shared-point slots: each slot used once, slots of a point in tile order
  std::vector<int> used(T.sh_ids.size(), 0), next(T.shp_off.begin(), T.shp_off.end() - 1);
  for (size_t k = 0; k < T.sh_ids.size(); ++k) {
    const int s = T.sh_ids[k] - T.shared_begin, slot = T.sh_slot[k];
    if (s < 0 || s >= T.nshared || slot != next[s]++ || used[slot]++) return -6;
  }
  for (int s = 0; s < T.nshared; ++s)
    if (next[s] != T.shp_off[s + 1] || T.shp_off[s + 1] - T.shp_off[s] < 2) return -6;
  out8[0] = T.ntiles;
  out8[1] = T.nshared;
  out8[2] = T.max_local;
  out8[3] = T.max_elems;
  out8[4] = max_col;
  out8[5] = nint;
  out8[6] = static_cast<long long>(T.sh_ids.size());
  // the tiles by rows of the same mesh: local ids, and phases in which no two
  // element classes add to one point
  Tiling U;
  if (!build_tiling(nspec, nglob, ibool, centroid_xz, tile_elems, U, nullptr, 1, nullptr, 1).empty()) return -1;
  out8[7] = 0;
  for (int t = 0; t < U.ntiles; ++t) {
    const TileInfo &ti = U.tiles[t];
    out8[7] = std::max<long long>(out8[7], ti.ncol);
    for (int p = 0; p < ti.ncol; ++p) {
      std::vector<char> mark(ti.n_int + ti.n_sh, 0);
      for (int s = ti.elem_base; s < ti.elem_base + ti.nelem; ++s) {
        const int e = U.elem_order[s];
        for (int q = 0; q < NGLL2; ++q) {
          const int l = U.lib[static_cast<size_t>(ti.lib_off) + static_cast<size_t>(s - ti.elem_base) * NGLL2 + q];
          if (U.glob_of(t, l) != ibool[static_cast<size_t>(e) * NGLL2 + q]) return -7;
          const int ph = (U.phases[s] >> (8 * phase_class(q))) & 127;
          if (ph >= ti.ncol || (ph == p && mark[l]++)) return -8;
        }
      }
    }
  }
  return 0;
}

// Host-side tiler: turns a reference-layout spectral-element mesh (ibool,
// per-element GLL arrays) into the tile-staged device layout.
//
// A tile is a set of up to `tile_elems` elements that one CTA advances per
// time step.  Its points are split into "interior" points (touched only by
// this tile's elements; stored contiguously in device numbering, owned and
// updated by the tile) and "shared" points (touched by several tiles, stored
// after all interior points and finished by a second kernel that adds the
// tiles' partial sums in tile order).  Shared points touched by the same tiles
// form a segment and are stored together, so that a tile's gathers and the
// second kernel's accesses are mostly contiguous.
//
// Two tile forms, one per element group:
// * coloured (the kernels that work on rows, columns and points of all the
//   tile's elements): elements are greedily coloured so that no two elements
//   of a colour share a point; shared-memory assembly runs colour by colour
//   without atomics.
// * by rows (the kernels with one element row per thread, five neighbouring
//   threads per element): elements stay in ascending order and a point's local
//   id follows (i, element, j), so that neighbouring threads read neighbouring
//   words of shared memory.  Assembly runs in phases over position classes
//   (phase_class): in a mesh whose elements have one orientation, no two
//   elements hold the same point at positions of one class, so four phases are
//   enough; elsewhere a class of an element moves to a later phase.
#pragma once

#include <cstdint>
#include <string>
#include <vector>

namespace sf2d {

constexpr int NGLL = 5;
constexpr int NGLL2 = 25;
constexpr int MAX_COLOURS = 8;
constexpr int MAX_PHASES = 100;  // phase numbers fit seven bits
constexpr int PHASE_CLASSES = 4;
// class of GLL position q = 5 j + i: 0 for i, j < 4, 1 for i = 4, j < 4, 2 for i < 4, j = 4, 3 for i = j = 4
constexpr int phase_class(int q) { return (q % 5 == 4 ? 1 : 0) + (q / 5 == 4 ? 2 : 0); }

struct TileInfo {
  int elem_base;   // first element slot of the tile (tile-ordered element arrays)
  int nelem;       // elements in the tile
  int n_int;       // interior local points
  int int_begin;   // device id of local point 0
  int n_sh;        // shared local points (local ids n_int .. n_int+n_sh-1)
  int sh_off;      // offset into sh_ids and sh_slot
  int st_off, st_n;    // boundary (Stacey) entries of this tile
  int src_off, src_n;  // source entries of this tile
  int rec_off, rec_n;  // receivers whose element lies in this tile
  int col_end[MAX_COLOURS];  // exclusive end (element index within tile) of each colour
  int ncol;        // colours, or assembly phases of a tile by rows
  int lib_off;     // offset of the tile's local ibool (multiple of 8 entries = 16 bytes)
  int cpl_off, cpl_n;  // fluid-solid coupling entries of this tile (none outside a coupled run)
  int edge_off, edge_n;  // local points on the outer edge of a CPML layer, zeroed every step
  int grp_off, grp_n;    // points that receive boundary, coupling or source terms (one thread each)
  int lane0;             // tile by rows: its first thread among all (a multiple of 32), five per element
};
static_assert(sizeof(TileInfo) == 29 * 4, "TileInfo layout");

struct Tiling {
  int ntiles = 0;
  int nglob = 0;
  int nelem = 0;
  int nshared = 0;       // number of shared points
  int shared_begin = 0;  // device id of the first shared point
  int max_local = 0;     // max local points over tiles
  int max_elems = 0;     // max elements over tiles
  std::vector<TileInfo> tiles;
  std::vector<int> elem_order;        // slot -> original element id
  std::vector<int> elem_tile;         // original element id -> tile
  std::vector<uint16_t> lib;          // lib_off + (slot - elem_base)*25 + q -> local point id
  std::vector<int> dev2glob;          // device id -> original global id
  std::vector<int> glob2dev;          // original global id -> device id
  std::vector<int> sh_ids;            // per tile shared local point -> device id
  std::vector<int> sh_slot;           // -> its partial-sum slot
  std::vector<int> shp_off;           // nshared+1: the slots of shared point s are [shp_off[s], shp_off[s+1]), tile order
  std::vector<uint32_t> phases;       // per slot of a tile by rows: phase of class k in byte k
  int nlanes = 0;                     // threads of all tiles by rows, each tile's rounded up to 32
  // local id of a global point in a tile, -1 when the tile does not hold it
  int local_id(int tile, int glob) const;
  // global point of a tile's local id
  int glob_of(int tile, int l) const {
    const TileInfo &t = tiles[tile];
    return dev2glob[l < t.n_int ? t.int_begin + l : sh_ids[t.sh_off + l - t.n_int]];
  }
  // tiles of element group k are [group_tile_begin[k], group_tile_begin[k+1])
  std::vector<int> group_tile_begin;
};

// Builds the tiling.  `ibool` is nspec*25 0-based ids in [ispec][j][i]
// order.  With `centroid_xz` (nspec*2, may be null) each group's elements are
// cut into compact tiles by recursive bisection, connected parts of the mesh
// (the members of a packed batch) one by one; without it they keep their
// input order.
// `elem_group` (nspec values in [0, ngroups), may be null) keeps elements of
// different groups in different tiles, group 0 first: the elements of a CPML
// layer get tiles (and a kernel variant) of their own.  `group_tile_elems`
// (ngroups values, may be null) sets a tile size per group; groups below
// `nlaned` get tiles by rows, the others coloured ones.
// Returns an empty string on success, else an error message.
std::string build_tiling(int nspec, int nglob, const int *ibool, const double *centroid_xz,
                         int tile_elems, Tiling &out, const int *elem_group = nullptr, int ngroups = 1,
                         const int *group_tile_elems = nullptr, int nlaned = 0);

}  // namespace sf2d

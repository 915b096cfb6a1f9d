// vlsg_frontier.cuh -- band passes that evaluate only the cells that can
// change.
//
// Every level-set buffer keeps, per allocated 8^3 brick, the values of all
// its cells (updated in place) and a 512-bit mask of its defined cells (one
// 64-bit word per z-plane, bit y*8+x).  A pass takes tiles of bricks, finds
// their candidate cells by bit dilation of the masks (neighbour
// bricks' face planes through the 27-neighbour table), evaluates the
// reference's rule on the candidates only and appends every (cell, new value)
// that changes to its warp's own segment of a change log (no atomics);
// kApplyChanges streams the log back afterwards, so every rule reads old values
// only -- the reference maps the whole old level set to a new one (Jacobi order).
// The new defined masks go to a second mask array.
// Candidates per pass:
//   Expand (lsExpand.hpp:104-157): undefined cells next to a defined one.  A
//     defined cell keeps its value when |v| <= width/2, which the engine
//     tracks per buffer; otherwise the defined cells are candidates too.
//     Without defined candidates the new values are written in place: see
//     kFrontierPass.
//   Prune (lsPrune.hpp:118-180): the defined cells (undefined ones keep their
//     sentinel).
//   rebuildLS (lsAdvect.hpp:299-415): defined cells and their neighbours (an
//     undefined cell with no defined neighbour keeps its sentinel).
//     After updateLevelSet the defined cells are the active ones (kUpdate).
// Bricks next to a boundary that remaps cells (reflective, periodic with a
// length that is not a multiple of 8, the mirrored side of POS/NEG_INFINITE)
// are "complex": neighbours outside the brick are read through the boundary
// mapping.
#pragma once

#include <cooperative_groups.h>

#include "vlsg_common.cuh"
#include "vlsg_passes.cuh"

namespace vlsg {
namespace { // internal linkage: every compilation unit has its own copy

constexpr int FRONTIER_THREADS = 256;
// Resident blocks per SM the passes are compiled for (40 registers per
// thread): the passes are bound by latency and issue, so occupancy pays more
// than the few spilled registers cost.
#ifndef VLSG_PASS_MIN_BLOCKS
#define VLSG_PASS_MIN_BLOCKS 6
#endif
constexpr uint64_t XLO = 0x0101010101010101ull; // cells with x = 0
constexpr uint64_t XHI = 0x8080808080808080ull; // cells with x = 7
// 27-neighbour table entries of the six faces (index (dz+1)*9+(dy+1)*3+dx+1)
constexpr int NB_XM = 12, NB_XP = 14, NB_YM = 10, NB_YP = 16, NB_ZM = 4, NB_ZP = 22;
constexpr uint8_t CF_STAR = 1; // a star neighbour of a cell is remapped
constexpr uint8_t CF_NEAR = 2; // a cell within 8 cells is remapped

// Brick topology shared by the passes.
struct Topo {
  GridDev g;
  const int *brickMap, *slotBrick, *slotList, *nSlots;
  const int *nbr;       // 27 entries per slot: slot, or -1-brick
  const uint8_t *cflag; // CF_* per slot
  int *err;
};

// Point data carried by the cells of the top level set (null arrays: none):
// the source id of the data a defined cell carries (the index of a point at
// the start of the advection, -1: none) and the saved advection velocity and
// dissipation (lsAdvect.hpp:780-796).  In a change log the same arrays hold
// the data of each logged cell.
template <class T> struct Payload {
  int32_t *src;
  T *vel, *diss;
};

template <class T> struct LsView {
  T *vals;               // slots x 512 cells, in place
  const uint64_t *def;   // current masks, slots x 8 words
  uint64_t *defNext;     // masks after the pass
  const int8_t *farSign; // per brick of the map box
  Payload<T> pd;         // point data per cell, or null arrays
  float *lo;             // compensation terms (FP32 buffers that carry them), or null
};

// Change log: segment w (of `per` entries) belongs to warp w of the pass.
template <class T> struct ChangeLog {
  uint32_t *cell; // slot << 9 | cell
  T *val;
  int *count;     // entries per segment
  size_t per;
  Payload<T> pd;  // point data per entry (with a view that carries it)
};

// Point data of the value a rule produced: src -1 keeps the centre's, 0..5
// takes star neighbour src's (cell loc of slot ref), -2 none.
template <class T>
__device__ inline void payloadOf(const Payload<T> &pd, size_t centre, int src, int ref, int loc,
                                 int32_t &s, T &v, T &d) {
  if (src == -1) {
    s = pd.src[centre], v = pd.vel[centre], d = pd.diss[centre];
  } else if (src >= 0 && ref >= 0) {
    const size_t q = (size_t)ref * BV + loc;
    s = pd.src[q], v = pd.vel[q], d = pd.diss[q];
  } else {
    s = -1, v = T(0), d = T(0);
  }
}

template <class T> __device__ inline T sentinel(bool neg) {
  return neg ? Lim<T>::lowest() : Lim<T>::max();
}

// Slot (or -1-brick) and cell index of global cell (x,y,z) through the
// boundary mapping; cells outside the map box take the nearest box cell.
__device__ inline int locateCell(const GridDev &g, const int *brickMap, int x, int y, int z,
                                 int &local) {
  x = mapCoord(g, 0, x), y = mapCoord(g, 1, y), z = mapCoord(g, 2, z);
  int rx = x - g.org[0], ry = y - g.org[1], rz = z - g.org[2];
  const int ex = g.nb[0] * BS - 1, ey = g.nb[1] * BS - 1, ez = g.nb[2] * BS - 1;
  rx = rx < 0 ? 0 : (rx > ex ? ex : rx);
  ry = ry < 0 ? 0 : (ry > ey ? ey : ry);
  rz = rz < 0 ? 0 : (rz > ez ? ez : rz);
  const int bi = brickIndex(g, rx >> 3, ry >> 3, rz >> 3);
  local = (rz & 7) * 64 + (ry & 7) * 8 + (rx & 7);
  const int slot = brickMap[bi];
  return slot >= 0 ? slot : -1 - bi;
}

// Face neighbours of a slot in the 27-table order -x,+x,-y,+y,-z,+z.
__device__ inline int faceEntry(int f) {
  return f == 0 ? NB_XM : f == 1 ? NB_XP : f == 2 ? NB_YM : f == 3 ? NB_YP : f == 4 ? NB_ZM : NB_ZP;
}

// Per-warp shared scratch of the brick in hand.
struct WarpScratch {
  unsigned long long flip[8]; // cells whose definedness flips
  uint16_t list[BV];          // the brick's cells to evaluate, ascending
};

__device__ inline void brickOrigin(const Topo &t, int slot, int &x0, int &y0, int &z0) {
  int bx, by, bz;
  brickCoords(t.g, t.slotBrick[slot], bx, by, bz);
  x0 = t.g.org[0] + bx * BS, y0 = t.g.org[1] + by * BS, z0 = t.g.org[2] + bz * BS;
}

// Star neighbour j (order +x,+y,+z,-x,-y,-z) of local cell c as (slot or
// -1-brick, cell): through the face neighbours, or, for a brick next to a
// boundary that remaps cells, through the brick map and the mapping.
__device__ inline int starRef(const Topo &t, const int *nb, int slot, bool complex, int x0,
                              int y0, int z0, int c, int j, int &loc) {
  const int x = c & 7, y = (c >> 3) & 7, z = c >> 6;
  if (complex) {
    const int dx = j == 0 ? 1 : j == 3 ? -1 : 0, dy = j == 1 ? 1 : j == 4 ? -1 : 0,
              dz = j == 2 ? 1 : j == 5 ? -1 : 0;
    const int nx = x + dx, ny = y + dy, nz = z + dz;
    if ((nx | ny | nz) >= 0 && (nx | ny | nz) < BS &&
        cellExists(t.g, x0 + nx, y0 + ny, z0 + nz)) {
      loc = nz * 64 + ny * 8 + nx;
      return slot;
    }
    return locateCell(t.g, t.brickMap, x0 + nx, y0 + ny, z0 + nz, loc);
  }
  switch (j) {
  case 0: loc = x < 7 ? c + 1 : c - 7; return x < 7 ? slot : nb[1];
  case 1: loc = y < 7 ? c + 8 : c - 56; return y < 7 ? slot : nb[3];
  case 2: loc = z < 7 ? c + 64 : c - 448; return z < 7 ? slot : nb[5];
  case 3: loc = x > 0 ? c - 1 : c + 7; return x > 0 ? slot : nb[0];
  case 4: loc = y > 0 ? c - 8 : c + 56; return y > 0 ? slot : nb[2];
  default: loc = z > 0 ? c - 64 : c + 448; return z > 0 ? slot : nb[4];
  }
}

// Local cells [lo, hi] of a brick starting at `base` that exist in direction d.
__device__ inline void existRange(const GridDev &g, int d, int base, int &lo, int &hi) {
  lo = 0, hi = BS - 1;
  const int bc = g.bc[d];
  if (bc == VLSG_PERIODIC_BOUNDARY || bc == VLSG_REFLECTIVE_BOUNDARY ||
      bc == VLSG_POS_INFINITE_BOUNDARY)
    lo = max(0, g.gmin[d] - base);
  if (bc == VLSG_PERIODIC_BOUNDARY || bc == VLSG_REFLECTIVE_BOUNDARY ||
      bc == VLSG_NEG_INFINITE_BOUNDARY)
    hi = min(BS - 1, g.gmax[d] - (bc == VLSG_PERIODIC_BOUNDARY ? 1 : 0) - base);
}
// Mask of the cells of plane z that exist in the grid.
__device__ inline uint64_t existPlane(const GridDev &g, int x0, int y0, int z0, int z) {
  int xl, xh, yl, yh, zl, zh;
  existRange(g, 0, x0, xl, xh);
  existRange(g, 1, y0, yl, yh);
  existRange(g, 2, z0, zl, zh);
  if (z < zl || z > zh || xl > xh || yl > yh) return 0ull;
  const uint64_t row = (0xffull << xl) & (0xffull >> (7 - xh)) & 0xffull;
  return row * XLO & (~0ull << (8 * yl)) & (~0ull >> (8 * (7 - yh)));
}

// List the set cells of a brick mask (lane z holds plane z, z < 8) into
// `list` in ascending order: lane l < 16 walks the 32-bit half l & 1 of plane
// l >> 1.  Returns the number of cells (every lane).  Every lane of the warp
// must call it.
__device__ inline int listCells(uint64_t plane, uint16_t *list) {
  const int lane = threadIdx.x & 31;
  const uint64_t pw = __shfl_sync(0xffffffffu, plane, lane >> 2);
  unsigned w = (unsigned)(pw >> (16 * (lane & 3))) & 0xffffu;
  const int cnt = __popc(w);
  int x = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += t;
  }
  int off = x - cnt;
  const int total = __shfl_sync(0xffffffffu, x, 31);
  const int base = (lane >> 2) * 64 + (lane & 3) * 16;
  while (w) {
    list[off++] = (uint16_t)(base + __ffs(w) - 1);
    w &= w - 1;
  }
  __syncwarp();
  return total;
}

__device__ inline void markCell(unsigned long long *words, int c) {
  // the 32-bit half of the plane word that holds the cell (little endian)
  atomicOr(reinterpret_cast<unsigned *>(words) + (c >> 5), 1u << (c & 31));
}

// Append the lanes with `has` to the warp's log segment (warp-uniform call),
// with the point data (ps, pv, pdi) when the log carries it.
template <class T>
__device__ inline void logChange(const ChangeLog<T> &lg, size_t base, int &count, bool has,
                                 uint32_t cell, T val, int32_t ps = -1, T pv = T(0),
                                 T pdi = T(0)) {
  const unsigned m = __ballot_sync(0xffffffffu, has);
  if (has) {
    const size_t p = base + count + __popc(m & ((1u << (threadIdx.x & 31)) - 1));
    lg.cell[p] = cell;
    lg.val[p] = val;
    if (lg.pd.src) lg.pd.src[p] = ps, lg.pd.vel[p] = pv, lg.pd.diss[p] = pdi;
  }
  count += __popc(m);
}

// A new value (and its point data) written in place; its compensation term
// becomes 0, as for every value a pass computes from stored values.
template <class T>
__device__ inline void putCell(const LsView<T> &v, size_t q, T out, bool data, int32_t ps, T pv,
                               T pdi) {
  if (data) v.pd.src[q] = ps, v.pd.vel[q] = pv, v.pd.diss[q] = pdi;
  v.vals[q] = out;
  if (v.lo) v.lo[q] = 0.f;
}

enum : int { FP_EXPAND = 0, FP_PRUNE = 1, FP_ALL = 2, FP_GROW = 3 };

// ---------------------------------------------------------------- brick tiles
//
// A pass works on tiles of up to 32 consecutive entries of the slot list, one
// tile per block of 256 threads at a time: the visited bricks' masks are
// dilated with one thread per brick plane, all candidate cells of the tile go
// into one list, and all threads take cells from it.  A warp per brick (about
// 90 candidates in the Expand passes of a sphere of 16.8M band points) left
// 40% of the lanes idle in the evaluation (19.5 of 32 active) and 24 of 32 in
// the mask work, and a small level set ran as long as one warp needs for a
// brick.  Few bricks: fewer per tile, so that every block has one.
// Measured, warp per brick -> tiles, one B200: Expand pass of that sphere 0.45
// -> 0.29 ms, rebuild 0.75 -> 0.59, Prune pair 0.60 -> 0.47; FP64 circle of 2000
// points (boundary path) Expand 29 -> 19 us; reflective FP64 trench, 101 x 75
// cells, Expand 78 -> 23 us (there the candidates now come from dilation too,
// not from every existing cell).
constexpr int TILE_BRICKS = 32;
constexpr int TILE_SCAN = 2;    // list entries per lane of the scan for visited bricks
constexpr int TILE_LIST = 4096; // cells listed at a time

struct TileScratch {
  int slot[TILE_BRICKS];
  int nb[TILE_BRICKS][6];          // face neighbours; -1 / -2: none, undefined + / -
  unsigned flip[TILE_BRICKS][16];  // cells whose definedness flips
  uint8_t map[TILE_BRICKS];        // brick next to a remapping boundary
  int sums[FRONTIER_THREADS / 32];
  int count, next;
  uint16_t list[TILE_LIST];        // brick of the tile << 9 | cell
};

// List entries per tile: equal shares of whole rounds of the grid, of at most 32
// entries; 64 from eight such rounds on (about 40% of the entries are visited
// bricks, of which a round takes 32).  Expand pass of the FP32 sphere of 16.8M
// points (600k entries): 0.29 ms with 32, 0.266 with 64; of the FP64 sphere of 2.2M
// (80k) 57 us with 32, 66 with 64, whose few tiles per block come out uneven.
__device__ inline int tileEntries(int n) {
  const int g = (int)gridDim.x;
  const int most = n >= 256 * g ? 32 * TILE_SCAN : 32;
  const int rounds = max(1, (n + g * most - 1) / (g * most));
  return max(1, (n + g * rounds - 1) / (g * rounds));
}

// Wrap position of a brick in direction d of a grid whose period is not a
// whole number of bricks: the last cell's local coordinate, seen from the
// first brick (`below`) and in the last one (`above`); 7 elsewhere.
__device__ inline void wrapCells(const GridDev &g, int d, int base, int &below, int &above) {
  below = above = BS - 1;
  if (g.bc[d] != VLSG_PERIODIC_BOUNDARY) return;
  const int last = (g.gmax[d] - 1 - g.gmin[d]) & (BS - 1);
  if (base <= g.gmin[d]) below = last;
  if (base + BS >= g.gmax[d]) above = last;
}

// Whether a mirroring wall lies at or within the lower (upper) face of a brick
// in direction d: past that face there are no cells of the grid.
__device__ inline bool mirrored(const GridDev &g, int d, int base, bool upper) {
  const int bc = g.bc[d];
  if (upper)
    return (bc == VLSG_REFLECTIVE_BOUNDARY || bc == VLSG_NEG_INFINITE_BOUNDARY) &&
           base + BS - 1 >= g.gmax[d];
  return (bc == VLSG_REFLECTIVE_BOUNDARY || bc == VLSG_POS_INFINITE_BOUNDARY) && base <= g.gmin[d];
}

// Star dilation of plane z of a brick's mask (w), in groups of 8 consecutive
// lanes of a warp, one per plane; nb: the brick's face neighbours.  Sets err
// bit 64 when a set cell lies on a face past which the grid goes on and whose
// neighbour brick is not allocated (its cells could change but are not in the
// pool).  map: the brick
// lies at a remapping boundary: planes and columns past a period's end are
// left out and the wrap takes the last existing ones; a mirrored neighbour is
// the opposite one, which the in-brick shifts already give.
template <bool MAP>
__device__ inline uint64_t dilateTile(const Topo &t, const uint64_t *mask, int slot, const int *nb,
                                      int z, uint64_t w, bool on, bool map) {
  uint64_t below = __shfl_sync(0xffffffffu, w, (z + 7) & 7, 8);
  uint64_t above = __shfl_sync(0xffffffffu, w, (z + 1) & 7, 8);
  if (!on) return 0ull;
  int px = 7, qx = 7, py = 7, qy = 7, pz = 7, qz = 7;
  uint64_t exist = ~0ull;
  if (MAP && map) {
    int x0, y0, z0;
    brickOrigin(t, slot, x0, y0, z0);
    wrapCells(t.g, 0, x0, px, qx);
    wrapCells(t.g, 1, y0, py, qy);
    wrapCells(t.g, 2, z0, pz, qz);
    exist = existPlane(t.g, x0, y0, z0, z);
    if (((w & XLO) && nb[0] < 0 && !mirrored(t.g, 0, x0, false)) ||
        (((w >> qx) & XLO) && nb[1] < 0 && !mirrored(t.g, 0, x0, true)) ||
        ((w & 0xffull) && nb[2] < 0 && !mirrored(t.g, 1, y0, false)) ||
        (((w >> (8 * qy)) & 0xffull) && nb[3] < 0 && !mirrored(t.g, 1, y0, true)) ||
        (z == 0 && w && nb[4] < 0 && !mirrored(t.g, 2, z0, false)) ||
        (z == qz && w && nb[5] < 0 && !mirrored(t.g, 2, z0, true)))
      atomicOr(t.err, 64);
  } else {
    const bool open = ((w & XLO) && nb[0] < 0) || ((w & XHI) && nb[1] < 0) ||
                      ((w & 0xffull) && nb[2] < 0) || ((w >> 56) && nb[3] < 0) ||
                      (z == 0 && w && nb[4] < 0) || (z == 7 && w && nb[5] < 0);
    if (open) atomicOr(t.err, 64);
  }
  const uint64_t nxm = nb[0] >= 0 ? mask[(size_t)nb[0] * 8 + z] : 0ull;
  const uint64_t nxp = nb[1] >= 0 ? mask[(size_t)nb[1] * 8 + z] : 0ull;
  const uint64_t nym = nb[2] >= 0 ? mask[(size_t)nb[2] * 8 + z] : 0ull;
  const uint64_t nyp = nb[3] >= 0 ? mask[(size_t)nb[3] * 8 + z] : 0ull;
  if (z == 0) below = nb[4] >= 0 ? mask[(size_t)nb[4] * 8 + pz] : 0ull;
  if (z == qz) above = nb[5] >= 0 ? mask[(size_t)nb[5] * 8] : 0ull;
  return exist & (w | ((w << 1) & ~XLO) | ((w >> 1) & ~XHI) | ((nxm >> px) & XLO) |
                  ((nxp & XLO) << qx) | (w << 8) | (w >> 8) | ((nym >> (8 * py)) & 0xffull) |
                  ((nyp & 0xffull) << (8 * qy)) | below | above);
}

// Exclusive scan of one count per thread of the block; *total: their sum.
// `sums`: shared, one per warp; the caller synchronises before its next use.
__device__ inline int tileScan(int *sums, int v, int *total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += u;
  }
  if (lane == 31) sums[wid] = x;
  __syncthreads();
  int before = 0, sum = 0;
#pragma unroll
  for (int k = 0; k < FRONTIER_THREADS / 32; ++k) {
    const int u = sums[k];
    before += k < wid ? u : 0;
    sum += u;
  }
  *total = sum;
  return before + x - v;
}

// Whether an undefined cell of brick `slot` (at a remapping boundary) has an
// undefined star neighbour of the other sign.  One warp: signs of the brick as
// planes (lane z < 8), from one read of it, then of the cells across its faces.
// nb: the face neighbours (TileScratch::nb).
template <class T>
__device__ inline bool oppositePairs(const Topo &t, const LsView<T> &v, int slot, const int *nb) {
  constexpr unsigned ALL = 0xffffffffu;
  const int lane = threadIdx.x & 31, z = lane & 7;
  int base[3], zl, zh;
  brickOrigin(t, slot, base[0], base[1], base[2]);
  existRange(t.g, 2, base[2], zl, zh);
  const uint64_t undef =
      existPlane(t.g, base[0], base[1], base[2], z) & ~v.def[(size_t)slot * 8 + z];
  uint64_t signs = 0ull; // set: negative
#pragma unroll 4
  for (int k = 2 * zl; k <= 2 * zh + 1; ++k) {
    const uint64_t b = __ballot_sync(ALL, v.vals[(size_t)slot * BV + 32 * k + lane] < T(0));
    if (z == k >> 1) signs |= b << (32 * (k & 1));
  }
  const uint64_t neg = undef & signs, pos = undef & ~signs;
  const uint64_t negUp = __shfl_sync(ALL, neg, (z + 1) & 7), posUp = __shfl_sync(ALL, pos, (z + 1) & 7);
  uint64_t hit = (pos & (neg >> 1) & ~XHI) | (neg & (pos >> 1) & ~XHI) | (pos & (neg >> 8)) |
                 (neg & (pos >> 8)) | (z < 7 ? (pos & negUp) | (neg & posUp) : 0ull);
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    const int d = f >> 1, r = nb[f];
    const bool upper = f & 1;
    if ((t.g.planar && d == 2) || mirrored(t.g, d, base[d], upper)) continue;
    int below, above;
    wrapCells(t.g, d, base[d], below, above);
    const int own = upper ? above : 0, other = upper ? 0 : below; // coordinates in d
    const uint64_t face = d == 0 ? XLO << own : d == 1 ? 0xffull << (8 * own) : z == own ? ~0ull : 0ull;
    if (r < 0) {
      hit |= face & (r == -2 ? pos : neg);
      continue;
    }
    // the neighbour's cells across the face (plane j >> 3, cell j & 7 of its row)
    uint64_t s = 0ull;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = 32 * h + lane;
      const int c = d == 0   ? (j >> 3) * 64 + (j & 7) * 8 + other
                    : d == 1 ? (j >> 3) * 64 + other * 8 + (j & 7)
                             : other * 64 + j;
      s |= (uint64_t)__ballot_sync(ALL, v.vals[(size_t)r * BV + c] < T(0)) << (32 * h);
    }
    // moved onto the face
    const uint64_t word = v.def[(size_t)r * 8 + (d == 2 ? other : z)];
    uint64_t sign = s, def = word;
    if (d == 0) {
      // bits 0..6 of the row to bits 0, 8, .., 48, bit 7 to 56
      const uint64_t row = (s >> (8 * z)) & 0xffull;
      sign = ((((row & 0x7full) * 0x0002040810204081ull) & XLO) | ((row >> 7) << 56)) << own;
      def = ((word >> other) & XLO) << own;
    } else if (d == 1) {
      sign = ((s >> (8 * z)) & 0xffull) << (8 * own);
      def = ((word >> (8 * other)) & 0xffull) << (8 * own);
    }
    hit |= face & ~def & ((pos & sign) | (neg & ~sign));
  }
  return __any_sync(ALL, hit != 0ull);
}

// Cell value through a resolved neighbour reference (TileScratch::nb).
template <class T> __device__ inline T tileValue(const T *vals, int ref, int loc) {
  return ref >= 0 ? vals[(size_t)ref * BV + loc] : sentinel<T>(ref == -2);
}

// FP_EXPAND passes write in place and may stand for two Expand cycles
// (expandStep, vlsg_expand.h, tells which and why).
//
// Let L be the limit of the pass.  A star neighbour that read a value v the
// pass defines would come to |v| + 1; v "feeds" when that is below L (in a pass
// of one cycle: L or below).  While no value feeds and none changes its cell's
// sign, a warp that sees another warp's store instead of the sentinel takes L
// or decides the same, so the pass needs no change log and no write-back; and
// two cycles (limits L - 1/2 and L) define what one pass with limit L defines,
// with the same values, but for cells of value L that are left to the next pass.
// A cell whose sign would change is not written.
// Either event sets *event, and kExpandRedo, launched after an Expand's passes,
// then does the whole Expand again, cycle by cycle: the passes have changed
// neither a value of the masks before them nor the sign of any cell.  It is one
// cluster of blocks; a host that has seen it work logs the next Expands instead
// (Engine::expandPart), on the whole GPU.  No event
// is missed: of two undefined cells of opposite sign side by side, the first to
// be evaluated sees the other's sign; a cell that becomes a candidate between
// the cycles of a pass is one in the next pass, and the last is a single cycle.
// Bands that miss cells within their width feed; bands whose undefined cells
// are of opposite sign side by side, or next to a value of the other sign of
// magnitude 1 or more, change signs.  In bricks at remapping boundaries a cycle
// takes every cell that it finds undefined, next to a defined one or not: there
// an Expand's first pass looks for all pairs of opposite sign (the later ones
// find no more, since cells only become defined).
// FP32 sphere of 16.8M points, per WENO5 + RK3 step: 19 passes and write-backs
// with one logged pass per cycle (8.6 + 2.2 ms), 16 passes now (4.3 ms).
//
// MODE picks the candidates: FP_EXPAND undefined cells next to a defined one,
// FP_GROW the same (logged), FP_PRUNE the defined cells, FP_ALL the defined
// cells and their neighbours; an Expand's logged passes also take the other
// cells of bricks at remapping boundaries.
// MAP: the grid has boundaries that remap cells.
// Returns, per thread, whether it met a defined +-0 (FP_PRUNE) or an event
// (FP_EXPAND, FP_GROW).
template <class T, int MODE, bool MAP, class Rule>
__device__ __forceinline__ bool frontierTiles(TileScratch &ts, const Topo &t, const LsView<T> &v,
                                              const Rule &rule, const ChangeLog<T> &lg,
                                              const uint8_t *visitIn, uint8_t *visitOut,
                                              bool wallPairs = false) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int warp = blockIdx.x * (FRONTIER_THREADS / 32) + wid;
  const int n = *t.nSlots;
  const size_t logBase = (size_t)warp * lg.per;
  int logged = 0;
  bool hit = false;
  const int per = tileEntries(n);
  const int tiles = (n + per - 1) / per;
  for (int tile = blockIdx.x, next = tile * per; tile < tiles;) {
    const int end = min((tile + 1) * per, n);
    if (wid == 0) {
      // the tile's bricks; one the previous pass of this buffer did not mark
      // has no defined cell and no defined face neighbour cell
      int slot[TILE_SCAN];
      bool in[TILE_SCAN], map[TILE_SCAN], go[TILE_SCAN];
#pragma unroll
      for (int k = 0; k < TILE_SCAN; ++k) {
        const int e = next + 32 * k + lane;
        in[k] = e < end;
        slot[k] = in[k] ? t.slotList[e] : 0;
      }
#pragma unroll
      for (int k = 0; k < TILE_SCAN; ++k) {
        map[k] = MAP && in[k] && (t.cflag[slot[k]] & CF_STAR) != 0;
        go[k] = in[k] && (!visitIn || map[k] || visitIn[slot[k]]);
      }
      int count = 0, stop = end;
#pragma unroll
      for (int k = 0; k < TILE_SCAN; ++k) {
        const unsigned mask = __ballot_sync(0xffffffffu, go[k]);
        const int p = count + __popc(mask & ((1u << lane) - 1));
        const unsigned over = __ballot_sync(0xffffffffu, go[k] && p >= TILE_BRICKS);
        if (over && stop == end) stop = next + 32 * k + __ffs(over) - 1; // the next round's first
        if (next + 32 * k + lane < stop) {
          if (go[k]) {
            ts.slot[p] = slot[k];
            if (MAP) ts.map[p] = map[k];
          } else if (in[k]) {
            uint4 *w = reinterpret_cast<uint4 *>(v.defNext + (size_t)slot[k] * 8);
            for (int j = 0; j < 4; ++j) w[j] = make_uint4(0u, 0u, 0u, 0u);
          }
        }
        count += __popc(mask);
      }
      if (lane == 0) ts.count = min(count, TILE_BRICKS), ts.next = stop;
    }
    __syncthreads();
    next = ts.next;
    // one thread per plane z of brick i: masks, candidates
    const int i = tid >> 3, z = tid & 7;
    const bool on = i < ts.count;
    const int slot = on ? ts.slot[i] : 0;
    const bool map = MAP && on && ts.map[i];
    const uint64_t own = on ? v.def[(size_t)slot * 8 + z] : 0ull;
    int face = -1;
    if (on) {
      ts.flip[i][2 * z] = ts.flip[i][2 * z + 1] = 0u;
      if (z < 6) {
        face = t.nbr[(size_t)slot * 27 + faceEntry(z)];
        if (face < 0) face = v.farSign[-1 - face] < 0 ? -2 : -1;
        ts.nb[i][z] = face;
      }
    }
    int nb[6];
#pragma unroll
    for (int f = 0; f < 6; ++f) nb[f] = __shfl_sync(0xffffffffu, face, f, 8);
    uint64_t cand = own;
    if (MODE != FP_PRUNE) {
      cand = dilateTile<MAP>(t, v.def, slot, nb, z, own, on, map);
      if (MAP && map && MODE != FP_EXPAND && Rule::wallCells) {
        int x0, y0, z0;
        brickOrigin(t, slot, x0, y0, z0);
        cand = existPlane(t.g, x0, y0, z0, z);
      }
      if (MODE == FP_EXPAND || MODE == FP_GROW) cand &= ~own;
    }
    int total;
    int at = tileScan(ts.sums, __popcll(cand), &total);
    if constexpr (MODE == FP_EXPAND && MAP) {
      if (wallPairs)
        for (int b = wid; b < ts.count; b += FRONTIER_THREADS / 32)
          if (ts.map[b]) hit |= oppositePairs<T>(t, v, ts.slot[b], ts.nb[b]);
    }
    for (int w0 = 0; w0 < total; w0 += TILE_LIST) {
      const int size = min(TILE_LIST, total - w0);
      while (cand && at < w0 + size) {
        ts.list[at++ - w0] = (uint16_t)((i << 9) | (z << 6) | (__ffsll((long long)cand) - 1));
        cand &= cand - 1;
      }
      __syncthreads();
      for (int base = 0; base < size; base += FRONTIER_THREADS) {
        const int k = base + tid;
        bool changed = false;
        T out = T(0);
        uint32_t cell = 0;
        int32_t ps = -1;
        T pv = T(0), pdi = T(0);
        if (k < size) {
          const int bi = ts.list[k] >> 9, c = ts.list[k] & (BV - 1);
          const int sl = ts.slot[bi];
          const bool mp = MAP && ts.map[bi];
          int x0 = 0, y0 = 0, z0 = 0;
          if (MAP && mp) brickOrigin(t, sl, x0, y0, z0);
          cell = ((uint32_t)sl << 9) | (uint32_t)c;
          const T center = v.vals[cell];
          if (MODE == FP_PRUNE && center == T(0)) hit = true;
          const auto ref = [&](int j, int &loc) {
            int r = starRef(t, ts.nb[bi], sl, MAP && mp, x0, y0, z0, c, j, loc);
            if (MAP && mp && r < 0) r = v.farSign[-1 - r] < 0 ? -2 : -1;
            return r;
          };
          T star[6];
#pragma unroll
          for (int j = 0; j < 6; ++j) {
            int loc;
            const int r = ref(j, loc);
            star[j] = tileValue<T>(v.vals, r, loc);
          }
          int src = -1;
          out = rule(center, star, src);
          changed = out != center || signbit(out) != signbit(center);
          if constexpr (MODE == FP_EXPAND || MODE == FP_GROW) {
            const bool turns = signbit(out) != signbit(center);
            hit |= turns || rule.feeds(center, out);
            if (MODE == FP_EXPAND && turns) changed = false;
          }
          if (changed && isDef(out) != isDef(center))
            atomicOr(&ts.flip[bi][c >> 5], 1u << (c & 31));
          // with point data a value taken from a neighbour is logged even when
          // it equals the old one: its data changes
          if (MODE != FP_EXPAND && lg.pd.src && isDef(out) && src >= 0) changed = true;
          if (changed && lg.pd.src && isDef(out)) {
            int loc = 0, r = -1;
            if (src >= 0) r = ref(src, loc);
            payloadOf<T>(v.pd, cell, src, r, loc, ps, pv, pdi);
          }
          if (MODE == FP_EXPAND && changed)
            putCell(v, cell, out, lg.pd.src != nullptr, ps, pv, pdi);
        }
        if (MODE != FP_EXPAND) logChange<T>(lg, logBase, logged, changed, cell, out, ps, pv, pdi);
      }
      __syncthreads();
    }
    // the new mask, and the bricks the next pass of this buffer must visit:
    // those with a defined cell, and each face neighbour of one with a defined
    // cell on the shared face (only those can have candidates)
    uint64_t nw = own;
    if (on) {
      nw ^= (uint64_t)ts.flip[i][2 * z] | ((uint64_t)ts.flip[i][2 * z + 1] << 32);
      v.defNext[(size_t)slot * 8 + z] = nw;
    }
    const int shift = lane & 24;
    const auto planes = [&](bool p) {
      return (__ballot_sync(0xffffffffu, on && p) >> shift) & 0xffu;
    };
    const unsigned any = planes(nw != 0ull), xm = planes((nw & XLO) != 0ull),
                   xp = planes((nw & XHI) != 0ull), ym = planes((nw & 0xffull) != 0ull),
                   yp = planes((nw >> 56) != 0ull);
    if (on && z < 7 && any) {
      const int f = z < 6 ? face : slot;
      const unsigned at = z == 0 ? xm : z == 1 ? xp : z == 2 ? ym : z == 3 ? yp
                          : z == 4 ? any & 1u : z == 5 ? any & 0x80u : 1u;
      if (at && f >= 0) visitOut[f] = 1;
    }
    __syncthreads();
    if (next >= end) tile += gridDim.x, next = tile * per;
  }
  if (MODE != FP_EXPAND && lane == 0) lg.count[warp] = logged;
  return hit;
}

template <class T, int MODE, bool MAP, class Rule>
__global__ void __launch_bounds__(FRONTIER_THREADS, VLSG_PASS_MIN_BLOCKS)
    kFrontierPass(Topo t, LsView<T> v, Rule rule, ChangeLog<T> lg, const uint8_t *visitIn,
                  uint8_t *visitOut, int *zeros, int zeroMode, int poolSlots, uint4 *clear,
                  size_t nClear, int *event) {
  __shared__ TileScratch ts;
  const int tid = threadIdx.x, lane = tid & 31;
  // the visit flags the next pass writes
  for (size_t k = (size_t)blockIdx.x * blockDim.x + tid; k < nClear;
       k += (size_t)gridDim.x * blockDim.x)
    clear[k] = make_uint4(0u, 0u, 0u, 0u);
  // zeroMode 1: record a defined candidate +-0 in *zeros; zeroMode 2: when
  // *zeros is 0 the pass is known to change nothing (the second Prune of a
  // pair): copy the masks and the visit flags of the whole pool (free slots
  // included, whose contents no one reads), log nothing; zeroMode 3 (FP_EXPAND):
  // look for opposite undefined cells at remapping boundaries (oppositePairs)
  if (MODE == FP_PRUNE && zeroMode == 2 && *zeros == 0) {
    const size_t first = (size_t)blockIdx.x * blockDim.x + tid;
    const size_t nThreads = (size_t)gridDim.x * blockDim.x;
    const uint4 *src = reinterpret_cast<const uint4 *>(v.def); // 4 x 16 bytes per slot
    uint4 *dst = reinterpret_cast<uint4 *>(v.defNext);
    for (size_t i = first; i < (size_t)poolSlots * 4; i += nThreads) dst[i] = src[i];
    if (visitOut)
      for (size_t i = first; i < (size_t)poolSlots; i += nThreads)
        visitOut[i] = visitIn ? visitIn[i] : 1;
    if (lane == 0) lg.count[(blockIdx.x * blockDim.x + tid) >> 5] = 0;
    return;
  }
  const bool hit = frontierTiles<T, MODE, MAP>(ts, t, v, rule, lg, visitIn, visitOut, zeroMode == 3);
  if (MODE == FP_PRUNE && zeroMode == 1 && __any_sync(0xffffffffu, hit) && lane == 0)
    atomicOr(zeros, 1);
  if ((MODE == FP_EXPAND || MODE == FP_GROW) && __any_sync(0xffffffffu, hit) && lane == 0)
    atomicOr(event, 1);
}

// Write segment w of a change log back: one warp, four loads in flight per lane.
// `lo` (FP32 buffers that carry a compensation term, else null): a cell a
// pass changed holds a value computed from the stored values alone, so its
// compensation term becomes 0.
template <class T>
__device__ inline void applySegment(T *vals, const ChangeLog<T> &lg, int w, float *lo,
                                    const Payload<T> &pd) {
  const int lane = threadIdx.x & 31;
  const int n = lg.count[w];
  const size_t base = (size_t)w * lg.per;
  for (int i = lane; i < n; i += 4 * 32) {
    uint32_t q[4];
    T val[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (i + 32 * k < n) q[k] = lg.cell[base + i + 32 * k], val[k] = lg.val[base + i + 32 * k];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (i + 32 * k < n) {
        vals[q[k]] = val[k];
        if (lo) lo[q[k]] = 0.f;
      }
  }
  // the point data the pass logged with each value
  if (pd.src && lg.pd.src)
    for (int i = lane; i < n; i += 32) {
      const uint32_t c = lg.cell[base + i];
      pd.src[c] = lg.pd.src[base + i];
      pd.vel[c] = lg.pd.vel[base + i];
      pd.diss[c] = lg.pd.diss[base + i];
    }
}
template <class T>
__global__ void __launch_bounds__(FRONTIER_THREADS)
    kApplyChanges(T *vals, ChangeLog<T> lg, int segments, float *lo, Payload<T> pd) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nWarps = (gridDim.x * blockDim.x) >> 5;
  for (int w = warp; w < segments; w += nWarps) applySegment(vals, lg, w, lo, pd);
}

// An Expand from width `at` (masks `from`) to `width` again, one logged cycle
// after another, if one of its FP_EXPAND passes met an event (kFrontierPass);
// else it returns at once.  `end`: the masks the passes left, which take the
// result; `mid`: a second array to alternate with; lg: a segment per warp of this
// kernel.  *seen tells the host.
// One cluster, whose blocks run together and have a barrier: a cooperative launch
// on the whole grid does so too, but waits for the other streams' kernels each
// time (48 domains of 1e4 to 1e6 points on 16 streams, LLF1 + RK2: 10.0 against
// 7.0 ms a step).
constexpr int REDO_BLOCKS = 8;
template <class T, class Rule>
__global__ void __cluster_dims__(REDO_BLOCKS, 1, 1) __launch_bounds__(FRONTIER_THREADS)
    kExpandRedo(Topo t, LsView<T> v, Rule rule, ChangeLog<T> lg, const uint64_t *from,
                uint64_t *end, uint64_t *mid, int at, int width, uint8_t *visit, int *event,
                int *seen) {
  if (*event == 0) return;
  __shared__ TileScratch ts;
  const cooperative_groups::cluster_group blocks = cooperative_groups::this_cluster();
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nWarps = (gridDim.x * blockDim.x) >> 5;
  const int n = *t.nSlots;
  // the cells the passes defined are undefined again, with their signs; every
  // brick is visited from here on
  for (int e = warp; e < n; e += nWarps) {
    const size_t slot = t.slotList[e];
    if (lane == 0) visit[slot] = 1;
    for (int k = 0; k < BV / 32; ++k) {
      const int c = 32 * k + lane;
      const uint64_t added = end[slot * 8 + (c >> 6)] & ~from[slot * 8 + (c >> 6)];
      T *p = v.vals + slot * BV + c;
      if ((added >> (c & 63)) & 1ull) *p = sentinel<T>(*p < 0);
    }
  }
  blocks.sync();
  for (int w = at + 1; w <= width; ++w) {
    v.def = w == at + 1 ? from : (width - w) & 1 ? end : mid;
    v.defNext = (width - w) & 1 ? mid : end;
    frontierTiles<T, FP_GROW, true>(ts, t, v, rule.cycle(w), lg, nullptr, visit);
    blocks.sync();
    applySegment(v.vals, lg, warp, v.lo, v.pd);
    blocks.sync();
  }
  if (blocks.thread_rank() == 0) *event = 0, *seen = 1;
}

// Pointwise boolean of two level sets, in place on A (booleanOpInternal,
// lsBooleanOperation.hpp:100-132); rewrites A's current masks.  `flag` is
// set when the comparator reports a move (combineLevelSets).
template <class T, class Comp>
__global__ void __launch_bounds__(FRONTIER_THREADS)
    kPointwise(Topo t, T *av, uint64_t *adef, const T *bv, Comp comp, int *flag, float *alo) {
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nWarps = (gridDim.x * blockDim.x) >> 5;
  const int n = *t.nSlots;
  for (int w = warp; w < n; w += nWarps) {
    const int slot = t.slotList[w];
    int bx, by, bz;
    brickCoords(t.g, t.slotBrick[slot], bx, by, bz);
    const int x0 = t.g.org[0] + bx * BS, y0 = t.g.org[1] + by * BS, z0 = t.g.org[2] + bz * BS;
    bool moved = false;
    uint64_t mine = 0;
    for (int z = 0; z < 8; ++z) {
      uint64_t bits = 0;
      for (int half = 0; half < 2; ++half) {
        const int c = z * 64 + half * 32 + lane;
        const size_t q = (size_t)slot * BV + c;
        const T a = av[q], bb = bv[q];
        bool mv = false;
        T o = comp(a, bb, mv);
        if (!cellExists(t.g, x0 + (c & 7), y0 + ((c >> 3) & 7), z0 + (c >> 6))) {
          o = Lim<T>::max();
          mv = false;
        }
        moved |= mv;
        if (o != a || signbit(o) != signbit(a)) {
          av[q] = o;
          if (alo) alo[q] = 0.f;
        }
        bits |= (uint64_t)__ballot_sync(0xffffffffu, isDef(o)) << (32 * half);
      }
      if (lane == z) mine = bits;
    }
    if (lane < 8) adef[(size_t)slot * 8 + lane] = mine;
    if (__any_sync(0xffffffffu, moved) && lane == 0 && flag) atomicOr(flag, 1);
  }
}

// Pointwise boolean for comparators that keep every undefined cell of A
// (combineLevelSets, lsAdvect.hpp:218-230): only A's defined cells are read,
// in place; A's masks lose the cells that became undefined.
// With compensation terms of both (FP32 buffers: alo for A, blo for B) the
// comparator sees hi + lo of each value in double and the result is split
// again into hi and lo (Comp::full); with alo alone a changed value's term
// becomes 0.
template <class T, class Comp>
__global__ void __launch_bounds__(FRONTIER_THREADS)
    kPointwiseDefined(Topo t, T *av, uint64_t *adef, const T *bv, Comp comp, int *flag,
                      float *alo, const float *blo) {
  __shared__ WarpScratch sm[FRONTIER_THREADS / 32];
  WarpScratch &ws = sm[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nWarps = (gridDim.x * blockDim.x) >> 5;
  const int n = *t.nSlots;
  bool moved = false;
  for (int w = warp; w < n; w += nWarps) {
    const int slot = t.slotList[w];
    const uint64_t own = lane < 8 ? adef[(size_t)slot * 8 + lane] : 0ull;
    if (!__any_sync(0xffffffffu, own != 0ull)) continue;
    if (lane < 8) ws.flip[lane] = 0ull;
    const int total = listCells(own, ws.list);
    for (int base = 0; base < total; base += 32) {
      const int k = base + lane;
      if (k >= total) continue;
      const int c = ws.list[k];
      const size_t q = (size_t)slot * BV + c;
      const T a = av[q];
      bool mv = false;
      if constexpr (sizeof(T) == 4) {
        if (alo && blo) {
          const T b = bv[q];
          if (isDef(b)) {
            const double r = comp.full(withLo((double)a, alo[q]), withLo((double)b, blo[q]), mv);
            const float hi = (float)r;
            av[q] = hi;
            alo[q] = (float)(r - (double)hi);
          } else {
            av[q] = b;
            markCell(ws.flip, c);
          }
          moved |= mv;
          continue;
        }
      }
      const T o = comp(a, bv[q], mv);
      moved |= mv;
      if (o != a || signbit(o) != signbit(a)) {
        av[q] = o;
        if (alo) alo[q] = 0.f;
        if (!isDef(o)) markCell(ws.flip, c);
      }
    }
    __syncwarp();
    if (lane < 8) adef[(size_t)slot * 8 + lane] = own & ~ws.flip[lane];
    __syncwarp();
  }
  if (__any_sync(0xffffffffu, moved) && lane == 0 && flag) atomicOr(flag, 1);
}

// Copy the listed slots of one buffer (values and masks) into another, 16
// bytes per thread.
// dlo (a compensation array of the destination, or null) receives slo, or
// zeros when the source has none.
template <class T>
__global__ void kCopySlots16(const int *slotList, const int *nSlots, const T *sv,
                             const uint64_t *sd, T *dv, uint64_t *dd, const float *slo,
                             float *dlo) {
  constexpr int PER = BV * sizeof(T) / 16; // 16-byte words per slot
  const size_t n = (size_t)*nSlots * PER;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const size_t slot = slotList[i / PER];
    const int k = (int)(i % PER);
    reinterpret_cast<uint4 *>(dv + slot * BV)[k] = reinterpret_cast<const uint4 *>(sv + slot * BV)[k];
    if (k < 4) reinterpret_cast<uint4 *>(dd + slot * 8)[k] = reinterpret_cast<const uint4 *>(sd + slot * 8)[k];
    if (dlo && k < BV * 4 / 16) {
      const uint4 z = make_uint4(0u, 0u, 0u, 0u);
      reinterpret_cast<uint4 *>(dlo + slot * BV)[k] =
          slo ? reinterpret_cast<const uint4 *>(slo + slot * BV)[k] : z;
    }
  }
}

// Neighbour table and complexity flags of every listed slot, for any
// boundary conditions: entry = slot, or -1-brick (unallocated, or outside the
// map box: the nearest box brick).  CF_STAR: the brick holds a cell whose
// star neighbour is remapped by a boundary (or a cell past the grid's end);
// CF_NEAR: such a cell lies within 8 cells of the brick.
__device__ inline bool remapNear(const GridDev &g, int d, int lo, int hi) {
  switch (g.bc[d]) {
  case VLSG_PERIODIC_BOUNDARY:
    return (g.gmax[d] - g.gmin[d]) % BS != 0 && (lo <= g.gmin[d] || hi >= g.gmax[d] - 1);
  case VLSG_REFLECTIVE_BOUNDARY:
    return lo <= g.gmin[d] || hi >= g.gmax[d];
  case VLSG_POS_INFINITE_BOUNDARY:
    return lo <= g.gmin[d];
  case VLSG_NEG_INFINITE_BOUNDARY:
    return hi >= g.gmax[d];
  default:
    return false;
  }
}

__global__ void kBuildNeighbours(GridDev g, const int *brickMap, const int *slotBrick,
                                 const int *slotList, const int *nSlots, int *nbr,
                                 uint8_t *cflag, int *slotDom) {
  const int n = *nSlots;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int slot = slotList[i];
    int bx, by, bz;
    brickCoords(g, slotBrick[slot], bx, by, bz);
    if (g.nDom) {
      // batching form: wrap within the brick's domain; a neighbour past the
      // domain's brick planes is the nearest plane's (unallocated) brick
      const int d = g.domOfBz[bz];
      slotDom[slot] = d;
      cflag[slot] = 0;
      for (int k = 0; k < 27; ++k) {
        int x = bx + k % 3 - 1, y = by + (k / 3) % 3 - 1, z = bz + k / 9 - 1;
        const bool inside = domainNeighbour(g, d, x, y, z);
        if (!inside) z = z < g.dom[d].bz0 ? g.dom[d].bz0 : g.dom[d].bz1 - 1;
        const int bi = brickIndex(g, x, y, z);
        const int s = brickMap[bi];
        nbr[(size_t)slot * 27 + k] = (s >= 0 && inside) ? s : -1 - bi;
      }
      continue;
    }
    const int bc[3] = {bx, by, bz};
    uint8_t f = 0;
    for (int d = 0; d < 3; ++d) {
      const int lo = g.org[d] + bc[d] * BS, hi = lo + BS - 1;
      if (remapNear(g, d, lo, hi)) f |= CF_STAR | CF_NEAR;
      if (remapNear(g, d, lo - BS, hi + BS)) f |= CF_NEAR;
    }
    cflag[slot] = f;
    for (int k = 0; k < 27; ++k) {
      int c[3] = {bx + k % 3 - 1, by + (k / 3) % 3 - 1, bz + k / 9 - 1};
      bool outside = false;
      for (int d = 0; d < 3; ++d) {
        if (c[d] >= 0 && c[d] < g.nb[d]) continue;
        if (g.bc[d] == VLSG_PERIODIC_BOUNDARY) {
          c[d] = (c[d] + g.nb[d]) % g.nb[d];
        } else {
          c[d] = c[d] < 0 ? 0 : g.nb[d] - 1;
          outside = true;
        }
      }
      const int bi = brickIndex(g, c[0], c[1], c[2]);
      const int s = brickMap[bi];
      nbr[(size_t)slot * 27 + k] = (s >= 0 && !outside) ? s : -1 - bi;
    }
  }
}

} // namespace
} // namespace vlsg

// Launch shape of the acoustic column kernels: host arithmetic alone (plain
// C++, so that the rule can be checked without a GPU).
#pragma once
#include <cstddef>
#include <initializer_list>

namespace wg {

// Block shape.  Timed (us per launch, 433 x 433 x 50 / 256 x 256 x 50 /
// 217 x 185 x 35 / 64 x 64 x 40): 16 columns x 26 lanes, 2 blocks per SM 619 /
// 220 / 93 / 16.9; 16 x 17, 2 blocks 619 / 229 / 94 / 17.4; 16 x 17, 3 blocks
// 630 / 223 / 99 / 19.5, 4 blocks 850 / 272 / 139 / 23.8 (56 registers spill);
// 16 x 13, 3 blocks 684 / 251 / 97 / 22; 32 x 17, 1 block 630 / 243 / 120 /
// 18.0; 32 x 26, 1 block 682 / 252 / 123 / 17.1; 32 x 32 761 / 276 / 137 / 18.8.
// Above 51 levels the lanes hold three or four levels and spill (52 and 196
// bytes per thread); against the 32 x 17 form still 422 -> 299 at 301 x 301 x 52,
// 731 -> 373 at 60 levels, 909 -> 580 at 80, 1090 -> 813 at 95.
#ifndef WG_COL_TY
#define WG_COL_TY 26
#endif
constexpr int COL_TY = WG_COL_TY;
constexpr int COL_NARR = 8;
constexpr int COL_NMET = 9;    // level coefficients staged per block ...
constexpr int COL_MET_NP = 4;  // ... for at most this many positions per lane
// The tallest column of the level-parallel kernel, at every width: what the
// shared memory of a 32-column block holds.
constexpr int COL_MAX_NZ = 112;
// Width of the default column kernel: 1 selects the one-thread-per-column
// streaming kernel (column_stream.cuh), 16 or 32 the level-parallel one
// (column_tiled.cuh).
#ifndef WG_COL_DEFAULT_WIDTH
#define WG_COL_DEFAULT_WIDTH 16
#endif
constexpr int COL_DEFAULT_WIDTH = WG_COL_DEFAULT_WIDTH;
static_assert(COL_DEFAULT_WIDTH == 1 || COL_DEFAULT_WIDTH == 16 || COL_DEFAULT_WIDTH == 32,
              "the default column width is 1, 16 or 32");
// Warps per block of the streaming kernel (each one row segment of 32
// columns); two blocks per SM.
#ifndef WG_CS_WARPS
#define WG_CS_WARPS 4
#endif
constexpr int CS_WARPS = WG_CS_WARPS;

inline size_t column_stream_smem_bytes(int nz) { return (size_t)2 * (nz + 1) * 32 * CS_WARPS * sizeof(double); }

inline size_t column_tiled_smem_bytes(int nz, int tx, int np) {
  return (size_t)(COL_NARR * tx + (np <= COL_MET_NP ? COL_NMET : 0)) * (nz + 1) * sizeof(double);
}

// Level lanes of a block and the positions per lane (np): the positions that the
// requested lanes, or COL_TY lanes, need -- at least 2 -- and then the fewest lanes that
// hold the column with them, so that all lanes end together.  A request that
// needs more than COL_MET_NP positions gets COL_TY lanes': beyond that the kernel
// spills hundreds of bytes per thread (us per launch, 160 x 150: 8 lanes, 7
// positions at nz = 50: 208, against 160 for the kernel with 8 whole lanes that
// the request used to name and 85 with 26; 13 lanes, 7 positions at nz = 80: 373,
// 311 and 156).  COL_TY lanes themselves reach 5 positions, above nz = 103.
constexpr int COL_MAX_NP = (COL_MAX_NZ + 1 + COL_TY - 1) / COL_TY;
inline int column_tiled_lanes(int nz, int tx, int lanes, int &np) {
  const int L = nz + 1, r0 = 32 / tx + 1;
  np = lanes > 0 ? (L + lanes - 1) / lanes : COL_MAX_NP;
  if (lanes <= 0 || np > COL_MET_NP) np = (L + COL_TY - 1) / COL_TY;
  if (np < 2) np = 2;
  const int ty = (L + np - 1) / np;
  return ty < r0 ? r0 : ty;
}

// The kernel and block for a requested column width (0: the default) and
// level-lane count (0: the default; the streaming kernel has none).
struct ColumnShape {
  bool stream;       // one thread per column
  int tx, ty, np;    // block (tx columns x ty lanes), positions per lane
  size_t smem;       // dynamic shared memory, bytes
  bool too_tall;     // more levels than the level-parallel kernel takes
};

inline ColumnShape column_shape(int nz, int width, int lanes) {
  ColumnShape s{};
  const int w = width > 0 ? width : COL_DEFAULT_WIDTH;
  s.stream = w == 1;
  if (s.stream) {
    s.tx = 32;
    s.ty = CS_WARPS;
    s.smem = column_stream_smem_bytes(nz);
    return s;
  }
  s.tx = w;
  s.too_tall = nz > COL_MAX_NZ;
  s.ty = column_tiled_lanes(nz, w, lanes, s.np);
  s.smem = column_tiled_smem_bytes(nz, w, s.np);
  return s;
}

// The column widths and lane counts the tuner tries at this height, each a
// different launch (lane counts that come to the same positions are one): the
// default first, then 32 columns and one thread per column.  Returns their number.
struct ColumnRequest {
  int width, lanes;
};
constexpr int COL_MAX_CANDIDATES = 7;

inline int column_candidates(int nz, ColumnRequest out[COL_MAX_CANDIDATES]) {
  int n = 0;
  for (int width : {16, 32, 1})
    for (int lanes : {0, 17, 13}) {
      const ColumnShape s = column_shape(nz, width, lanes);
      bool seen = false;
      for (int k = 0; k < n; ++k) {
        const ColumnShape t = column_shape(nz, out[k].width, out[k].lanes);
        seen = seen || (s.stream == t.stream && s.tx == t.tx && s.ty == t.ty && s.np == t.np);
      }
      if (!seen) out[n++] = {width, lanes};
    }
  return n;
}

}  // namespace wg

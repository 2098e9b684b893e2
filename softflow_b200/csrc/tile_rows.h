// tile_rows.h -- force tiles and the tile rows a marker's stencil reaches
// (plain C++: also compiled on the host by the tests).
#pragma once

#ifdef __CUDACC__
#define SFG_HD __host__ __device__
#else
#define SFG_HD
#endif

namespace sfg {

// Force-tile geometry.
constexpr int TILE_W = 32;
constexpr int TILE_H = 8;
constexpr int TILE_CELLS = TILE_W * TILE_H;

// Tile rows of the first and last of a stencil's rows iy0 - 1 .. iy0 + 2, both
// inside the lattice of ny rows wherever the marker lies: a valid marker's rows
// may begin at ny (a channel periodic in y, or a marker placed above it), where
// (iy0 - 1) / TILE_H is past the last tile row when ny is a multiple of TILE_H.
SFG_HD constexpr int row_inside(int iy, int ny) { return iy < 0 ? 0 : (iy < ny ? iy : ny - 1); }
SFG_HD constexpr int first_tile_row(int iy0, int ny) { return row_inside(iy0 - 1, ny) / TILE_H; }
SFG_HD constexpr int last_tile_row(int iy0, int ny) { return row_inside(iy0 + 2, ny) / TILE_H; }

}  // namespace sfg

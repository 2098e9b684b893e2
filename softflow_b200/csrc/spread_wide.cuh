// spread_wide.cuh -- ordered accumulation of 4 x 4 stencils into a force tile
// (FP64: the spreads of the step and of sfg_spread_forces), in the reference's
// serial order and without atomics.
//
// A tile's markers are applied in ascending order, the reference's loop order; its
// list is sorted once (tile_list_sort), and later sweeps of a step find it so.
// Markers are staged WIDE_CHUNK at a time, four lanes per marker, one stencil row
// each: a point's contribution and accumulator index go into the slot of the lane
// that owns its cell.  Lane (a, b) = (lane & 7, lane >> 3) owns the cells of columns
// a mod 8 and rows b mod 4: a stencil has 4 consecutive columns and rows, so its
// points fall on distinct lanes.  Then every lane adds its own point of each marker
// to its own cell, marker after marker, so every cell receives its terms in list
// order.
//
// A warp takes a whole tile, or a band of eight columns of it, four warps (a CTA)
// the tile; for its band it picks the entries of the list whose stencil reaches it,
// about a third.  Where one tile holds both sides of the periodic seam
// (nx <= TILE_W) two stencil columns can share a residue mod 8, but not a band, so a
// warp with a whole tile takes its four bands one after the other.
//
// A tile's markers are one serial chain; with one warp for the whole tile the
// longest list was the kernel's length (500 rings of 40 markers on 1000 x 700:
// 55 us for lists of 7 on average).
#pragma once
#include <climits>

#include "common.cuh"

namespace sfg {

constexpr int BAND_W = 8;                         // columns of a band
constexpr int BAND_WARPS = TILE_W / BAND_W;       // warps of a CTA, one per band
constexpr int WIDE_CHUNK = 8;
constexpr int SORT_LIST = 256;                    // entries sorted in shared memory
constexpr int SORT_SMEM = 2 * SORT_LIST;          // and the ints that takes

// A warp's accumulators, LIST entries picked at a time and a staged chunk.  Rows of
// W + 4 cells: the stencil points (4 rows x 4 columns) then fall on 16 distinct bank
// pairs; the four padding columns x 8 rows give every lane a cell of its own for
// markers it has no point of.
template <int W, int LIST>
struct BandSmem {
    static constexpr int ROW = W + 4, CELLS = TILE_H * ROW, PICKS = LIST;
    double ax[CELLS], ay[CELLS];
    double2 v[WIDE_CHUNK][33];                 // [marker][owner lane] (padded row)
    unsigned short cell[WIDE_CHUNK][32];       // accumulator index of that point
    unsigned mask[WIDE_CHUNK];                 // owner lanes holding a point
    int list[LIST];                            // picked entries (markers)
};
using BandTile = BandSmem<BAND_W, 256>;        // one of a CTA's four warps
using WarpTile = BandSmem<TILE_W, 32>;         // a warp with a whole tile

// One value a lane, ascending over the warp.
__device__ __forceinline__ int warp_sort(int v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            const int o = __shfl_xor_sync(0xffffffffu, v, j);
            const bool take_min = ((lane & j) == 0) == ((lane & k) == 0);
            v = take_min ? min(v, o) : max(v, o);
        }
    return v;
}

template <int THREADS>
__device__ __forceinline__ void group_sync() {
    if constexpr (THREADS == 32) __syncwarp(); else __syncthreads();
}

// a[0 .. n - 1] ascending, by the THREADS of a warp or CTA (t: this one): a bitonic
// merge sort whose comparisons all leave the smaller value below (each merge begins
// by comparing mirrored places), so that places from n on need not exist.
template <int THREADS>
__device__ __forceinline__ void group_sort(int* a, int n, int t) {
    int lg = 0;
    while ((1 << lg) < n) ++lg;
    auto step = [&](auto place) {
        for (int i = t; i < (1 << lg) / 2; i += THREADS) {
            const int2 p = place(i);
            if (p.y < n) {
                const int x = a[p.x], y = a[p.y];
                if (x > y) {
                    a[p.x] = y;
                    a[p.y] = x;
                }
            }
        }
        group_sync<THREADS>();
    };
    for (int k = 1; k <= lg; ++k) {
        const int h = 1 << (k - 1);
        step([&](int i) {
            const int lo = (i >> (k - 1) << k) + (i & (h - 1));
            return make_int2(lo, lo ^ ((1 << k) - 1));
        });
        for (int j = k - 2; j >= 0; --j)
            step([&](int i) {
                const int lo = (i >> j << (j + 1)) + (i & ((1 << j) - 1));
                return make_int2(lo, lo + (1 << j));
            });
    }
}

// Sorts a tile's list in place (one of at most 32 entries only where `keep` asks for
// it) and returns the calling lane's entry of its first 32.  All THREADS of the group
// call it; `smem` holds SORT_SMEM ints, aligned to 16 bytes.
template <int THREADS>
__device__ __forceinline__ int tile_list_sort(int* list, int cnt, int* smem, int t, bool keep) {
    const int lane = threadIdx.x & 31;
    if (cnt <= 32) {
        const int v = warp_sort(lane < cnt ? list[lane] : INT_MAX);
        if (keep) {
            group_sync<THREADS>();             // (every warp has read the list)
            if (t < cnt) list[t] = v;
            if constexpr (THREADS == 32) __syncwarp();
        }
        return v;
    }
    group_sync<THREADS>();                     // (the last tile's entries have been read)
    if (cnt <= SORT_LIST) {                    // by counting the entries below each
        int* sorted = smem + SORT_LIST;
        const int quads = (cnt + 3) / 4;
        for (int i = t; i < 4 * quads; i += THREADS) smem[i] = i < cnt ? list[i] : INT_MAX;
        group_sync<THREADS>();
        for (int i = t; i < cnt; i += THREADS) {
            const int v = smem[i];
            int rank = 0;
#pragma unroll 4
            for (int q = 0; q < quads; ++q) {
                const int4 o = reinterpret_cast<const int4*>(smem)[q];
                rank += (o.x < v) + (o.y < v) + (o.z < v) + (o.w < v);
            }
            sorted[rank] = v;
            list[rank] = v;
        }
        group_sync<THREADS>();
        return sorted[lane];
    }
    group_sort<THREADS>(list, cnt, t);
    return list[lane];
}

// The stencil data one staging lane needs: the marker's force and arc length, its
// origin, the four column weights and the weight of the lane's row.
struct BandMarker {
    double2 f;
    double ds, wx[4], wy;
    int2 org;
};

// Adds the contributions (f w) ds, in the reference's rounding order, of a tile's
// markers (a sorted list, `first` the lane's entry of its first 32) to the warp's
// accumulators.  PICK: to those of the band of eight columns from x0, in the
// accumulators from column `col` on, else to all of the tile's, from column x0.
// `y0`: first row of the tile.  org_of(m): stencil origin; load(m, sy, k): the
// marker's data for stencil row sy.
template <bool PICK, typename Smem, typename OrgOf, typename Load>
__device__ __forceinline__ void band_spread(Smem& B, const int* list, int cnt, int first, int nx,
                                            int ny, int x0, int col, int y0, int lane, OrgOf org_of,
                                            Load load) {
    constexpr int W = PICK ? BAND_W : TILE_W, ROW = Smem::ROW;
    const int pad = (lane >> 2) * ROW + (ROW - 4) + (lane & 3);   // this lane's padding cell
    const int jm = lane >> 2, sy = lane & 3;
    auto column = [&](int ox, int k) {
        int jx = ox - 1 + k;
        if (jx < 0) jx += nx;
        if (jx >= nx) jx -= nx;
        return jx;
    };
    for (int at = 0; at < cnt; at += PICK ? Smem::PICKS : cnt) {
        int n = cnt;
        if constexpr (PICK) {
            const int part = min(Smem::PICKS, cnt - at);
            n = 0;
            for (int i = 0; i < part; i += 32) {
                int m = 0;
                bool hit = false;
                if (i + lane < part) {
                    m = at + i == 0 ? first : list[at + i + lane];
                    const int ox = org_of(m).x;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int jx = column(ox, k);
                        hit = hit || (jx >= x0 && jx < x0 + W && jx >= 0 && jx < nx);
                    }
                }
                const unsigned b = __ballot_sync(0xffffffffu, hit);
                if (hit) B.list[n + __popc(b & ((1u << lane) - 1u))] = m;
                n += __popc(b);
            }
            __syncwarp();
        }
        auto entry = [&](int k) { return PICK ? B.list[k] : list[k]; };
        BandMarker k{};
        if (jm < n) load(entry(jm), sy, k);
        for (int c0 = 0; c0 < n; c0 += WIDE_CHUNK) {
            const int nb = min(WIDE_CHUNK, n - c0);
            __syncwarp();
            unsigned bits = 0u;
            const int iy = k.org.y - 1 + sy, cyl = iy - y0;
            const bool ok = !(isnan(k.f.x) || isnan(k.f.y));
            if (jm < nb && ok && cyl >= 0 && cyl < TILE_H && iy >= 0 && iy < ny) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int jx = column(k.org.x, q), cl = jx - x0;
                    const double w = k.wx[q] * k.wy;
                    if (cl >= 0 && cl < W && jx >= 0 && jx < nx && w > 1e-15) {
                        const int t = (cl & 7) + 8 * (cyl & 3);
                        B.v[jm][t] = make_double2(k.f.x * w * k.ds, k.f.y * w * k.ds);
                        B.cell[jm][t] = (unsigned short)(cyl * ROW + col + cl);
                        bits |= 1u << t;
                    }
                }
            }
            bits |= __shfl_xor_sync(0xffffffffu, bits, 1);
            bits |= __shfl_xor_sync(0xffffffffu, bits, 2);
            if (sy == 0 && jm < nb) B.mask[jm] = bits;
            __syncwarp();
            // the next chunk's data is in flight while this one is added
            if (c0 + WIDE_CHUNK + jm < n) load(entry(c0 + WIDE_CHUNK + jm), sy, k);
            // this lane's point of marker j (or zero into its padding cell, so
            // that the additions carry no branches)
            auto point = [&](int j, int& c, double2& v) {
                const bool h = (B.mask[j] >> lane) & 1u;
                const int ci = B.cell[j][lane];
                const double2 vi = B.v[j][lane];
                c = h ? ci : pad;
                v = h ? vi : make_double2(0.0, 0.0);
            };
            int j = 0;
            // two markers at a time: both cells are read before either is
            // written, the second addition taking the first's sum when both
            // points are the same cell (same order, same rounding)
            for (; j + 1 < nb; j += 2) {
                int c0i, c1i;
                double2 v0, v1;
                point(j, c0i, v0);
                point(j + 1, c1i, v1);
                double a0x = B.ax[c0i], a0y = B.ay[c0i];
                double a1x = B.ax[c1i], a1y = B.ay[c1i];
                a0x += v0.x;
                a0y += v0.y;
                B.ax[c0i] = a0x;
                B.ay[c0i] = a0y;
                const bool same = c1i == c0i;
                a1x = same ? a0x : a1x;
                a1y = same ? a0y : a1y;
                B.ax[c1i] = a1x + v1.x;
                B.ay[c1i] = a1y + v1.y;
            }
            if (j < nb) {
                int c;
                double2 v;
                point(j, c, v);
                B.ax[c] += v.x;
                B.ay[c] += v.y;
            }
        }
        __syncwarp();
    }
}

}  // namespace sfg

// spread_wide.cuh -- ordered accumulation of 4 x 4 stencils into a force tile
// (FP64: the spreads of the step and of sfg_spread_forces), in the reference's
// serial order and without atomics.
//
// One warp takes a band of eight columns of a 32 x 8 tile, four warps (a CTA) the
// tile.  A warp first picks the entries of the tile's marker list whose stencil
// reaches its band (about a third) and sorts those by marker, the reference's
// loop order.  Lane (a, b) = (lane & 7, lane >> 3) owns the band's cells of column
// a and rows b, b + 4; a stencil has 4 consecutive columns and rows, so its points
// in the band fall on distinct lanes, whatever the channel's width.  Markers are
// staged WIDE_CHUNK at a time, four lanes per marker, one stencil row each: a
// point's contribution and accumulator index go into the slot of the lane that
// owns its cell.  Then every lane adds its own point of each marker to its own
// cell, marker after marker, so every cell receives its terms in list order.
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
// Rows of 12 cells: the stencil points (4 rows x 4 columns) then fall on 16
// distinct bank pairs; four padding columns x 8 rows give every lane a cell of
// its own for markers it has no point of.
constexpr int BAND_ACC_W = BAND_W + 4;
constexpr int BAND_ACC = TILE_H * BAND_ACC_W;
constexpr int BAND_LIST = 256;   // entries sorted in shared memory (a power of two:
                                 // the bitonic sort pads to one)
constexpr int WIDE_CHUNK = 8;

struct BandSmem {
    double ax[BAND_ACC], ay[BAND_ACC];
    int list[BAND_LIST];                       // the band's entries (markers)
    double2 v[WIDE_CHUNK][33];                 // [marker][owner lane] (padded row)
    unsigned short cell[WIDE_CHUNK][32];       // accumulator index of that point
    unsigned mask[WIDE_CHUNK];                 // owner lanes holding a point
};

// Sorts cnt <= BAND_LIST markers in shared memory, ascending, by one warp.
__device__ __forceinline__ void band_sort(int* a, int cnt, int lane) {
    if (cnt <= 32) {
        // bitonic sort across the warp's registers (ascending by lane)
        int v = lane < cnt ? a[lane] : INT_MAX;
#pragma unroll
        for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
            for (int j = k >> 1; j > 0; j >>= 1) {
                const int o = __shfl_xor_sync(0xffffffffu, v, j);
                const bool take_min = ((lane & j) == 0) == ((lane & k) == 0);
                v = take_min ? min(v, o) : max(v, o);
            }
        if (lane < cnt) a[lane] = v;
    } else {
        int pow2 = 64;
        while (pow2 < cnt) pow2 <<= 1;
        for (int i = cnt + lane; i < pow2; i += 32) a[i] = INT_MAX;
        __syncwarp();
        for (int k = 2; k <= pow2; k <<= 1)
            for (int j = k >> 1; j > 0; j >>= 1) {
                for (int i = lane; i < pow2; i += 32) {
                    const int l = i ^ j;
                    if (l > i) {
                        const int x = a[i], y = a[l];
                        if ((x > y) == ((i & k) == 0)) { a[i] = y; a[l] = x; }
                    }
                }
                __syncwarp();
            }
    }
    __syncwarp();
}

// Sorts a list longer than BAND_LIST in place, by one thread (rare).
__device__ __forceinline__ void long_list_sort(int* a, int cnt) {
    for (int i = 1; i < cnt; ++i) {
        const int v = a[i];
        int j = i - 1;
        while (j >= 0 && a[j] > v) { a[j + 1] = a[j]; --j; }
        a[j + 1] = v;
    }
}

// The stencil data one staging lane needs: the marker's force and arc length, its
// origin, the four column weights and the weight of the lane's row.
struct BandMarker {
    double2 f;
    double ds, wx[4], wy;
    int2 org;
};

// Adds the contributions (f w) ds, in the reference's rounding order, of a tile's
// markers to the warp's accumulators.  `x0`: first column of the band, `y0`:
// first row of the tile.  org_of(m): stencil origin; load(m, sy, k): the marker's
// data for stencil row sy.  Lists longer than BAND_LIST are already sorted.
template <typename OrgOf, typename Load>
__device__ __forceinline__ void band_spread(BandSmem& B, const int* list, int cnt,
                                            int nx, int ny, int x0, int y0, int lane, OrgOf org_of,
                                            Load load) {
    const int pad = (lane >> 2) * BAND_ACC_W + BAND_W + (lane & 3);   // this lane's padding cell
    const int jm = lane >> 2, sy = lane & 3;
    auto column = [&](int ox, int k) {
        int jx = ox - 1 + k;
        if (jx < 0) jx += nx;
        if (jx >= nx) jx -= nx;
        return jx;
    };
    for (int at = 0; at < cnt; at += BAND_LIST) {
        const int part = min(BAND_LIST, cnt - at);
        int n = 0;
        for (int i = 0; i < part; i += 32) {
            int m = 0;
            bool hit = false;
            if (i + lane < part) {
                m = list[at + i + lane];
                const int ox = org_of(m).x;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int jx = column(ox, k);
                    hit = hit || (jx >= x0 && jx < x0 + BAND_W && jx >= 0 && jx < nx);
                }
            }
            const unsigned b = __ballot_sync(0xffffffffu, hit);
            if (hit) B.list[n + __popc(b & ((1u << lane) - 1u))] = m;
            n += __popc(b);
        }
        __syncwarp();
        if (cnt <= BAND_LIST) band_sort(B.list, n, lane);
        BandMarker k{};
        if (jm < n) load(B.list[jm], sy, k);
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
                    if (cl >= 0 && cl < BAND_W && jx >= 0 && jx < nx && w > 1e-15) {
                        const int t = cl + 8 * (cyl & 3);
                        B.v[jm][t] = make_double2(k.f.x * w * k.ds, k.f.y * w * k.ds);
                        B.cell[jm][t] = (unsigned short)(cyl * BAND_ACC_W + cl);
                        bits |= 1u << t;
                    }
                }
            }
            bits |= __shfl_xor_sync(0xffffffffu, bits, 1);
            bits |= __shfl_xor_sync(0xffffffffu, bits, 2);
            if (sy == 0 && jm < nb) B.mask[jm] = bits;
            __syncwarp();
            // the next chunk's data is in flight while this one is added
            if (c0 + WIDE_CHUNK + jm < n) load(B.list[c0 + WIDE_CHUNK + jm], sy, k);
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

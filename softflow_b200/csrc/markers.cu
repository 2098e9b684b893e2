// markers.cu -- marker-side kernels (FP64, compiled with --fmad=false).
//
// Membrane mechanics follow reference src/membrane/capsule.cpp:149-671,
// contact follows src/membrane/repulsion.cpp:6-284 with the cell list of
// src/membrane/cell_list.h:36-146, and the immersed-boundary coupling
// follows src/coupling/immersed_boundary.cpp:25-286.
//
// Spreading is a deterministic gather: every lattice cell of a touched
// 32 x 8 force tile sums the contributions of the markers whose 4 x 4
// stencil covers it, in ascending marker order (the reference's serial
// order), with no floating-point atomics.
#include <climits>

#include "markers.cuh"
#include "lattice.cuh"
#include "sfg_internal.h"
#include "ibm_interp.cuh"
#include "launch.cuh"
#include "spread_wide.cuh"

namespace sfg {

// ============================ membrane forces ==============================
// One warp per capsule.  Nodes are staged in shared memory; lanes work on
// nodes/edges in parallel; the ring reductions (area, perimeter) run
// sequentially in lane 0 in the reference's order.  Each node applies the
// contributions of its two edges (or three bending stencils) in the order
// in which the reference's edge loop reaches them.

constexpr int MEM_WARPS = 4;
constexpr int MEM_DOUBLES_PER_NODE = 11;  // P, F, E, GN, GP (2 each) + OK

__device__ __forceinline__ void apply_edges(double2* F, const double2* E, const double* OK, int n,
                                            int k, double s_first, double s_second) {
    // node k is the first node of edge k and the second node of edge k-1
    double2 a = F[k];
    if (k == 0) {
        if (OK[0] != 0.0) { a.x = a.x + s_first * E[0].x; a.y = a.y + s_first * E[0].y; }
        if (n > 1 && OK[n - 1] != 0.0) {
            a.x = a.x + s_second * E[n - 1].x;
            a.y = a.y + s_second * E[n - 1].y;
        }
    } else {
        if (OK[k - 1] != 0.0) {
            a.x = a.x + s_second * E[k - 1].x;
            a.y = a.y + s_second * E[k - 1].y;
        }
        if (OK[k] != 0.0) { a.x = a.x + s_first * E[k].x; a.y = a.y + s_first * E[k].y; }
    }
    F[k] = a;
}
// s_first / s_second are +1 or -1: multiplying by them is exact, so
// a + (-1) * e == a - e bit for bit.

__global__ void k_membrane(const CapsuleDev* __restrict__ caps, int ncaps, MarkerBufs mb,
                           int* __restrict__ has_prev, int maxn, unsigned* status) {
    extern __shared__ double smem[];
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int c = blockIdx.x * MEM_WARPS + warp;
    if (c >= ncaps) return;
    double* base = smem + (size_t)warp * MEM_DOUBLES_PER_NODE * maxn;
    double2* P = reinterpret_cast<double2*>(base);
    double2* F = P + maxn;
    double2* E = F + maxn;
    double2* GN = E + maxn;
    double2* GP = GN + maxn;
    double* OK = reinterpret_cast<double*>(GP + maxn);
    const CapsuleDev cp = caps[c];
    const int n = cp.n, off = cp.off;
    if (n > maxn) {
        if (lane == 0) atomicOr(status, (unsigned)ST_CAPSULE_TOO_BIG);
        return;
    }
    const double Lx = (double)cp.periodic_nx;
    for (int k = lane; k < n; k += 32) {
        P[k] = mb.pos[off + k];
        F[k] = make_double2(0.0, 0.0);
    }
    __syncwarp();

    // ---- stretching (capsule.cpp:338-470) ----
    for (int i = lane; i < n; i += 32) {
        const int j = (i + 1) % n;
        const double2 diff = min_image_d(P[j], P[i], Lx);
        const double L = norm_d(diff);
        if (L < 1e-15) { OK[i] = 0.0; continue; }
        const double L0 = mb.rest_len[off + i];
        double F_mag;
        if (cp.model == 1) {            // Neo-Hookean
            double lambda = L / L0;
            double inv3 = 1.0 / (lambda * lambda * lambda);
            F_mag = cp.G_s * (lambda - inv3);
        } else if (cp.model == 2) {     // Skalak
            double lambda = L / L0;
            double l2 = lambda * lambda;
            F_mag = cp.G_s * lambda * (l2 - 1.0) * (1.0 + cp.C_skalak);
        } else if (cp.model == 3) {     // WLC + power-law repulsion
            double L_max = cp.wlc_L_max_ratio * L0;
            double x = L / L_max;
            if (x > 0.99) x = 0.99;
            double F_wlc = cp.wlc_kBT_p * (1.0 / (4.0 * (1.0 - x) * (1.0 - x)) - 0.25 + x);
            double F_pow = -cp.wlc_k_pow / L;
            F_mag = F_wlc + F_pow;
        } else {                        // Hookean
            F_mag = cp.k_stretch * (L / L0 - 1.0);
        }
        const double2 dir = make_double2(diff.x / L, diff.y / L);
        E[i] = make_double2(dir.x * F_mag, dir.y * F_mag);
        OK[i] = 1.0;
    }
    __syncwarp();
    for (int k = lane; k < n; k += 32) apply_edges(F, E, OK, n, k, 1.0, -1.0);
    __syncwarp();

    // ---- bending (capsule.cpp:476-541) ----
    if (cp.use_helfrich) {
        for (int i = lane; i < n; i += 32) {
            const int ip = (i - 1 + n) % n, in = (i + 1) % n;
            const double2 ep = min_image_d(P[i], P[ip], Lx);
            const double2 en = min_image_d(P[in], P[i], Lx);
            const double lp2 = ep.x * ep.x + ep.y * ep.y, ln2 = en.x * en.x + en.y * en.y;
            if (lp2 < 1e-30 || ln2 < 1e-30) { OK[i] = 0.0; continue; }
            const double dth = atan2(ep.x * en.y - ep.y * en.x, ep.x * en.x + ep.y * en.y) -
                               mb.rest_ang[off + i];
            const double cc = -cp.k_bend * dth / mb.rest_ds[off + i];
            const double2 gn = make_double2(-en.y / ln2, en.x / ln2);
            const double2 gp = make_double2(-ep.y / lp2, ep.x / lp2);
            GN[i] = make_double2(gn.x * cc, gn.y * cc);
            GP[i] = make_double2(gp.x * cc, gp.y * cc);
            E[i] = make_double2((gn.x + gp.x) * cc, (gn.y + gp.y) * cc);
            OK[i] = 1.0;
        }
        __syncwarp();
        for (int k = lane; k < n; k += 32) {
            // stencils i in {k-1, k, k+1} touch node k; apply in loop order
            int ids[3] = {(k - 1 + n) % n, k, (k + 1) % n};
            for (int a = 0; a < 3; ++a)
                for (int b = a + 1; b < 3; ++b)
                    if (ids[b] < ids[a]) { int t = ids[a]; ids[a] = ids[b]; ids[b] = t; }
            double2 acc = F[k];
            for (int a = 0; a < 3; ++a) {
                const int i = ids[a];
                if (a > 0 && i == ids[a - 1]) continue;
                if (OK[i] == 0.0) continue;
                if ((i + 1) % n == k) { acc.x = acc.x + GN[i].x; acc.y = acc.y + GN[i].y; }
                if ((i - 1 + n) % n == k) { acc.x = acc.x + GP[i].x; acc.y = acc.y + GP[i].y; }
                if (i == k) { acc.x = acc.x - E[i].x; acc.y = acc.y - E[i].y; }
            }
            F[k] = acc;
        }
    } else {
        for (int i = lane; i < n; i += 32) {
            const double2 dp = min_image_d(P[(i - 1 + n) % n], P[i], Lx);
            const double2 dn = min_image_d(P[(i + 1) % n], P[i], Lx);
            const double2 lap = make_double2(dp.x + dn.x, dp.y + dn.y);
            F[i] = make_double2(F[i].x + lap.x * cp.k_bend, F[i].y + lap.y * cp.k_bend);
        }
    }
    __syncwarp();

    // ---- ring reductions in the reference's order (capsule.cpp:175-204) ----
    // The per-edge terms (minimum-image edge vector, edge length) are formed
    // by the lanes in parallel, with the same expressions; lane 0 then sums
    // them in the reference's order, so the sums are the same bit for bit.
    for (int i = lane; i < n; i += 32) {
        const double2 d = min_image_d(P[(i + 1) % n], P[i], Lx);
        GN[i] = d;
        E[i].x = norm_d(d);
    }
    __syncwarp();
    double sarea = 0.0, perim = 0.0;
    if (lane == 0) {
        if (Lx > 0.0) {
            double2 cur = P[0];
            for (int i = 0; i < n; ++i) {
                double2 nxt;
                if (i + 1 < n) {
                    const double2 d = GN[i];
                    nxt = make_double2(cur.x + d.x, cur.y + d.y);
                } else {
                    nxt = P[0];
                }
                sarea += cur.x * nxt.y - cur.y * nxt.x;
                cur = nxt;
            }
        } else {
            for (int i = 0; i < n; ++i) {
                const double2 a = P[i], b = P[(i + 1) % n];
                sarea += a.x * b.y - a.y * b.x;
            }
        }
        for (int i = 0; i < n; ++i) perim += E[i].x;
    }
    sarea = __shfl_sync(0xffffffffu, sarea, 0);
    perim = __shfl_sync(0xffffffffu, perim, 0);

    // ---- area penalty (capsule.cpp:547-586) ----
    {
        const double A = 0.5 * fabs(sarea), A0 = cp.rest_area;
        if (!(A0 < 1e-15)) {
            const double coeff = -cp.k_area * (A - A0) / A0;
            const double sign = (sarea >= 0.0) ? 1.0 : -1.0;
            for (int i = lane; i < n; i += 32) {
                const double2 ep = min_image_d(P[i], P[(i - 1 + n) % n], Lx);
                const double2 en = min_image_d(P[(i + 1) % n], P[i], Lx);
                double2 o = make_double2((ep.y + en.y) * 0.5, (-ep.x + -en.x) * 0.5);
                const double len = norm_d(o);
                if (len < 1e-15) continue;
                o = make_double2(o.x / len * sign, o.y / len * sign);
                F[i] = make_double2(F[i].x + o.x * coeff, F[i].y + o.y * coeff);
            }
        }
    }
    __syncwarp();

    // ---- perimeter penalty (capsule.cpp:588-604) ----
    {
        const double P0 = cp.rest_perimeter;
        if (!(P0 < 1e-15)) {
            const double coeff = -cp.k_perimeter * (perim - P0) / P0;
            for (int i = lane; i < n; i += 32) {
                const double2 diff = min_image_d(P[(i + 1) % n], P[i], Lx);
                const double L = norm_d(diff);
                if (L < 1e-15) { OK[i] = 0.0; continue; }
                E[i] = make_double2(diff.x / L * coeff, diff.y / L * coeff);
                OK[i] = 1.0;
            }
            __syncwarp();
            for (int k = lane; k < n; k += 32) apply_edges(F, E, OK, n, k, -1.0, 1.0);
            __syncwarp();
        }
    }

    // ---- lab-frame damping (capsule.cpp:606-610) ----
    for (int k = lane; k < n; k += 32) {
        const double2 v = mb.vel[off + k];
        F[k] = make_double2(F[k].x - v.x * cp.gamma_visc, F[k].y - v.y * cp.gamma_visc);
    }
    __syncwarp();

    // ---- Kelvin-Voigt membrane viscosity (capsule.cpp:612-671) ----
    if (cp.eta_membrane > 0.0) {
        if (!has_prev[c]) {
            for (int i = lane; i < n; i += 32)
                mb.prev_len[off + i] = norm_d(min_image_d(P[(i + 1) % n], P[i], Lx));
            __syncwarp();
            if (lane == 0) has_prev[c] = 1;
        } else {
            for (int i = lane; i < n; i += 32) {
                const double2 diff = min_image_d(P[(i + 1) % n], P[i], Lx);
                const double L = norm_d(diff);
                if (L < 1e-15) { OK[i] = 0.0; continue; }
                const double strain = (L - mb.prev_len[off + i]) / mb.rest_len[off + i];
                const double Fv = cp.eta_membrane * strain;
                E[i] = make_double2(diff.x / L * Fv, diff.y / L * Fv);
                OK[i] = 1.0;
                mb.prev_len[off + i] = L;
            }
            __syncwarp();
            for (int k = lane; k < n; k += 32) apply_edges(F, E, OK, n, k, 1.0, -1.0);
            __syncwarp();
        }
    }
    for (int k = lane; k < n; k += 32) mb.frc[off + k] = F[k];
}

// ================================ contact ==================================

__device__ __forceinline__ int contact_cell(const ChannelDev& ch, double2 p) {
    if (!finite2(p)) return 0;
    const double Lx = (double)ch.nx;
    double px = p.x - 0.0;
    px = fmod(px, Lx);
    if (px < 0.0) px += Lx;
    int cx = (int)floor(px / ch.cdx);
    int cy = (int)floor((p.y - ch.y_bot) / ch.cdy);
    if (cx < 0) cx = 0;
    if (cx >= ch.ncx) cx = ch.ncx - 1;
    if (cy < 0) cy = 0;
    if (cy >= ch.ncy) cy = ch.ncy - 1;
    return cy * ch.ncx + cx;
}

__device__ __forceinline__ double2 pair_force(const ChannelDev& ch, double2 pa, double2 va,
                                              double2 pb, double2 vb) {
    const double Lx = (double)ch.nx;
    double2 diff = make_double2(pa.x - pb.x, pa.y - pb.y);
    if (Lx > 0.0) {
        if (diff.x > 0.5 * Lx) diff.x -= Lx;
        if (diff.x < -0.5 * Lx) diff.x += Lx;
    }
    // far pairs without the square root: beyond r_cut^2 by more than its rounding,
    // r >= r_cut follows (an infinite r_cut^2 rejects nothing)
    if (diff.x * diff.x + diff.y * diff.y > ch.rep_r_cut * ch.rep_r_cut * (1.0 + 1e-14))
        return make_double2(0.0, 0.0);
    const double r = norm_d(diff);
    if (r < 1e-15 || r >= ch.rep_r_cut) return make_double2(0.0, 0.0);
    const double2 nrm = make_double2(diff.x / r, diff.y / r);
    const double F_rep = ch.rep_epsilon * pow(ch.rep_sigma / r, (double)ch.rep_power);
    double F_n = F_rep;
    double2 F_t = make_double2(0.0, 0.0);
    if (ch.rep_damping > 0.0 || ch.rep_friction > 0.0) {
        const double2 vr = make_double2(va.x - vb.x, va.y - vb.y);
        const double v_n = vr.x * nrm.x + vr.y * nrm.y;
        F_n = F_rep - ch.rep_damping * v_n;
        if (F_n < 0.0) F_n = 0.0;
        if (ch.rep_friction > 0.0) {
            const double2 vt = make_double2(vr.x - nrm.x * v_n, vr.y - nrm.y * v_n);
            const double vtm = norm_d(vt);
            if (vtm > 1e-12) {
                const double s = -ch.rep_friction * F_n;
                F_t = make_double2(vt.x / vtm * s, vt.y / vtm * s);
            }
        }
    }
    return make_double2(nrm.x * F_n + F_t.x, nrm.y * F_n + F_t.y);
}

// The cell list without a scan: k_marker_prep pushes every marker onto its
// cell's linked list (the cell's head, ContactBufs::next by marker); here the marker
// that reached its empty cell first walks that list, takes list space for the
// cell (one atomic per warp), sorts the cell's markers into the reference's
// insertion order (capsule-major, node-minor = ascending marker index) and
// replaces the cell's record by (start, count).  Where a cell's markers lie
// in the list does not matter, only their order within the cell.  The work
// follows the markers instead of the cells (5 to 20 times as many), and the
// records of visited cells are cleared again by the marker move, so nothing
// runs over all cells: on 30 capsules the binning, three-kernel scan, fill
// and sort with their two memsets were nine graph nodes in a row.
//
// Up to CONTACT_BUF markers one thread sorts in its own memory; a more crowded cell
// (fine membranes, a long cut-off) is ranked by its warp.  By one thread the lists
// phase of 7,000 markers with cells of 30 to 250 took 84 to 721 us, so 29 to 54.
constexpr int CONTACT_BUF = 12;
__device__ __forceinline__ void contact_cells(int m, int M, const ChannelDev* __restrict__ chans,
                                              const MarkerBufs& mb, const ContactBufs& cb,
                                              int* total) {
    bool owner = m < M;
    int c = 0, n = 0, head = 0;
    int buf[CONTACT_BUF];
    if (owner) {
        owner = !chans[mb.mk_chan[m]].brute_contact && cb.next[m] == 0;
        if (owner) {
            c = cb.cell_of[m];
            head = cb.cell[c].x;
            for (int i = head; i != 0; i = cb.next[i - 1]) {
                if (n < CONTACT_BUF) buf[n] = i - 1;
                ++n;
            }
        }
    }
    const int lane = threadIdx.x & 31;
    int inc = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    int base = 0;
    if (lane == 31 && inc > 0) base = atomicAdd(total, inc);
    base = __shfl_sync(0xffffffffu, base, 31) + inc - n;
    if (owner) cb.cell[c] = make_int2(base, n);
    if (owner && n <= CONTACT_BUF) {
        for (int i = 1; i < n; ++i) {
            const int v = buf[i];
            int j = i - 1;
            while (j >= 0 && buf[j] > v) { buf[j + 1] = buf[j]; --j; }
            buf[j + 1] = v;
        }
        for (int i = 0; i < n; ++i) {
            cb.list[base + i] = make_int2(buf[i], mb.mk_cap[buf[i]]);
            cb.lpos[base + i] = mb.pos[buf[i]];
        }
    }
    // crowded cells, one after the other by the whole warp: the owner has left the
    // markers as they came in the memory of the cell's positions, every lane counts
    // how many precede its own
    const bool crowded = owner && n > CONTACT_BUF;
    if (crowded) {
        int* came = reinterpret_cast<int*>(cb.lpos + base);
        for (int i = head, k = 0; i != 0; i = cb.next[i - 1], ++k) came[k] = i - 1;
    }
    __syncwarp();
    for (unsigned left = __ballot_sync(0xffffffffu, crowded); left; left &= left - 1) {
        const int o = __ffs(left) - 1;
        const int at = __shfl_sync(0xffffffffu, base, o), cnt = __shfl_sync(0xffffffffu, n, o);
        const int* came = reinterpret_cast<const int*>(cb.lpos + at);
        for (int e = lane; e < cnt; e += 32) {
            const int v = came[e];
            int rank = 0;
#pragma unroll 8
            for (int k = 0; k < cnt; ++k) rank += came[k] < v ? 1 : 0;
            cb.list[at + rank] = make_int2(v, mb.mk_cap[v]);
        }
        __syncwarp();
        for (int e = lane; e < cnt; e += 32) cb.lpos[at + e] = mb.pos[cb.list[at + e].x];
        __syncwarp();
    }
}

// List entries of a cell loaded at once (nearly all are of the marker's own
// capsule, and one by one each waited for its load: contact phase of 720 markers
// 16.1 us one by one, 15.0 by four, 14.9 by eight; a step of 12 ragged channels 89.4,
// 88.7, 87.7, of 256 channels 499, 494, 492).
constexpr int CONTACT_AHEAD = 8;

// The cells k0 .. k1 - 1 of a marker's 3 x 3 neighbourhood, row by row (x in
// [0, ncx) wrapped, rows outside empty).  One after the other in a loop that is not
// unrolled, the next record loaded ahead: nine copies of the pair force did not
// stay in the instruction cache (516,096 markers with a cut-off of 14: contact phase
// 1,373 us with nine copies, 1,081 so; 7,000 markers 401 -> 233).
struct ContactCells {
    int cx, cy, k0, k1;
    __device__ __forceinline__ ContactCells(const ChannelDev& ch, const ContactBufs& cb, int m,
                                            int first, int end)
        : k0(first), k1(end) {
        const int ci = cb.cell_of[m] - ch.cell_base;
        cx = ci % ch.ncx;
        cy = ci / ch.ncx;
    }
    __device__ __forceinline__ int2 rec(const ChannelDev& ch, const ContactBufs& cb, int k) const {
        const int yy = cy + k / 3 - 1;
        int xx = cx + k % 3 - 1;
        if (xx < 0) xx += ch.ncx;
        if (xx >= ch.ncx) xx -= ch.ncx;
        return k >= k1 || yy < 0 || yy >= ch.ncy ? make_int2(0, 0)
                                                 : cb.cell[ch.cell_base + yy * ch.ncx + xx];
    }
    // add(f) for every marker of another capsule, in the cells' order, until it
    // returns false; an entry of the same capsule costs one 8-byte load, another
    // capsule's entry also the position copied into the list.  Velocities are
    // read only where damping or friction use them.
    template <typename Add>
    __device__ __forceinline__ void each(const ChannelDev& ch, const MarkerBufs& mb,
                                         const ContactBufs& cb, int cap, double2 pa, double2 va,
                                         Add add) const {
        const bool moving = ch.rep_damping > 0.0 || ch.rep_friction > 0.0;
        int2 next = rec(ch, cb, k0);
#pragma unroll 1
        for (int k = k0; k < k1; ++k) {
            const int2 now = next;
            next = rec(ch, cb, k + 1);
            const int end = now.x + now.y;
            for (int e0 = now.x; e0 < end; e0 += CONTACT_AHEAD) {
                // list entries are (marker, capsule)
                unsigned others = 0;
#pragma unroll
                for (int j = 0; j < CONTACT_AHEAD; ++j)
                    if (cb.list[min(e0 + j, end - 1)].y != cap && e0 + j < end) others |= 1u << j;
                for (; others; others &= others - 1) {
                    const int e = e0 + __ffs(others) - 1;
                    if (!add(pair_force(ch, pa, va, cb.lpos[e],
                                        moving ? mb.vel[cb.list[e].x] : make_double2(0.0, 0.0))))
                        return;
                }
            }
        }
    }
};

__device__ __forceinline__ void add2(double2& F, double2 f) {
    F.x = F.x + f.x;
    F.y = F.y + f.y;
}

// The whole of a marker's contact force by one thread.
__device__ __forceinline__ int contact_serial(const ChannelDev& ch, const MarkerBufs& mb,
                                              const ContactBufs& cb, int m, int cap, double2 pa,
                                              double2 va, double2& F) {
    int count = 0;
    if (ch.brute_contact) {
        for (int b = ch.mk_begin; b < ch.mk_end; ++b) {
            if (mb.mk_cap[b] == cap) continue;
            add2(F, pair_force(ch, pa, va, mb.pos[b], mb.vel[b]));
            ++count;
        }
    } else {
        ContactCells(ch, cb, m, 0, 9).each(ch, mb, cb, cap, pa, va, [&](double2 f) {
            add2(F, f);
            ++count;
            return true;
        });
    }
    return count;
}

// Contact and wall forces of a marker, by one thread or (QUAD) by four lanes,
// which take two or three of the nine cells each and a wall each.  The forces
// that are not zero (a few at most, as the cut-off is below the cells' width)
// are kept by the lanes and added in the cells' order by all four, so the sum
// is the one thread's; a lane that finds more than QUAD_PAIRS of them leaves
// the marker to one thread.  By interp_by_quads: with 720 to 2400 markers
// 17.1 -> 15.4 us, with two capsules in the cell-free form 19.1 -> 14.9; with
// 72,000 markers 18.9 -> 35.1 and 204,528 30.4 -> 85.9, whose chip is full.
// A lane that has found more stops there, as the one thread counts them anew.  One
// thread a marker is bound by the latency of dependent FP64 instructions: three
// blocks resident (80 registers) where 88 registers kept two; 516,096 markers with
// a cut-off of 14 1,312 -> 1,081 us.
constexpr int QUAD_PAIRS = 4;
template <bool QUAD>
__global__ void __launch_bounds__(256, QUAD ? 2 : 3)
k_contact_force(const ChannelDev* __restrict__ chans, int M, MarkerBufs mb, ContactBufs cb) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, m = QUAD ? t >> 2 : t;
    if (!QUAD && m >= M) return;
    const bool on = m < M;   // (lanes beyond the last marker only take part)
    const ChannelDev& ch = chans[on ? mb.mk_chan[m] : 0];
    const int cap = on ? mb.mk_cap[m] : 0;
    const double2 z = make_double2(0.0, 0.0);
    const double2 pa = on ? mb.pos[m] : z, va = on ? mb.vel[m] : z;
    double2 F = on ? mb.frc[m] : z;
    const double2 bot = make_double2(pa.x, ch.y_bot), top = make_double2(pa.x, ch.y_top);
    if constexpr (!QUAD) {
        const int count = contact_serial(ch, mb, cb, m, cap, pa, va, F);
        add2(F, pair_force(ch, pa, va, bot, z));
        add2(F, pair_force(ch, pa, va, top, z));
        mb.frc[m] = F;
        mb.pair_count[m] = count;
    } else {
        const int q = t & 3;
        double2 keep[QUAD_PAIRS];
#pragma unroll
        for (int i = 0; i < QUAD_PAIRS; ++i) keep[i] = z;
        int n = 0, count = 0;
        if (on && !ch.brute_contact) {
            ContactCells(ch, cb, m, q == 0 ? 0 : 2 * q + 1, 2 * q + 3)
                .each(ch, mb, cb, cap, pa, va, [&](double2 f) {
                    ++count;
                    if (f.x == 0.0 && f.y == 0.0) return true;
#pragma unroll
                    for (int i = 0; i < QUAD_PAIRS; ++i)
                        if (i == n) keep[i] = f;
                    return ++n <= QUAD_PAIRS;
                });
        }
        const double2 wall = pair_force(ch, pa, va, (q & 1) ? top : bot, z);
        int most = n;
        most = max(most, __shfl_xor_sync(0xffffffffu, most, 1));
        most = max(most, __shfl_xor_sync(0xffffffffu, most, 2));
        count += __shfl_xor_sync(0xffffffffu, count, 1);
        count += __shfl_xor_sync(0xffffffffu, count, 2);
        const bool serial = on && (ch.brute_contact || most > QUAD_PAIRS);
        if (serial && q == 0) count = contact_serial(ch, mb, cb, m, cap, pa, va, F);
        if (count > 0 && !serial) add2(F, z);   // (the zero forces: -0 becomes +0)
        for (int l = 0; l < 4; ++l) {
            const int got = __shfl_sync(0xffffffffu, n, l, 4), nl = serial ? 0 : got;
#pragma unroll
            for (int i = 0; i < QUAD_PAIRS; ++i) {
                if (!__any_sync(0xffffffffu, i < nl)) break;   // uniform in the warp
                const double fx = __shfl_sync(0xffffffffu, keep[i].x, l, 4);
                const double fy = __shfl_sync(0xffffffffu, keep[i].y, l, 4);
                if (i < nl) add2(F, make_double2(fx, fy));
            }
        }
        const double tx = __shfl_sync(0xffffffffu, wall.x, 1, 4);
        const double ty = __shfl_sync(0xffffffffu, wall.y, 1, 4);
        if (!on || q != 0) return;
        add2(F, wall);
        add2(F, make_double2(tx, ty));
        mb.frc[m] = F;
        mb.pair_count[m] = count;
    }
}

// ====================== immersed-boundary force tiles ======================

// Tiles covered by the stencil of a marker (at most 4 columns x 2 rows).
__device__ __forceinline__ int stencil_tiles(const ChannelDev& ch, int ix0, int iy0, int out[8]) {
    int tys[2], nty = 0;
    for (int iy = iy0 - 1; iy <= iy0 + 2; ++iy) {
        if (iy < 0 || iy >= ch.ny) continue;
        const int ty = iy / TILE_H;
        if (nty == 0 || tys[nty - 1] != ty) tys[nty++] = ty;
    }
    int txs[4], ntx = 0;
    for (int ix = ix0 - 1; ix <= ix0 + 2; ++ix) {
        int jx = ix;
        if (jx < 0) jx += ch.nx;
        if (jx >= ch.nx) jx -= ch.nx;
        if (jx < 0 || jx >= ch.nx) continue;
        const int tx = jx / TILE_W;
        bool dup = false;
        for (int a = 0; a < ntx; ++a) dup |= (txs[a] == tx);
        if (!dup) txs[ntx++] = tx;
    }
    int n = 0;
    for (int a = 0; a < nty; ++a)
        for (int b = 0; b < ntx; ++b) out[n++] = ch.tile_base + tys[a] * ch.tiles_x + txs[b];
    return n;
}

// Counts (FILL false) or list places (true) of a marker's stencil tiles among
// the lanes of a warp that share them: one atomic per distinct tile and warp.
// All lanes of the warp call it, lanes without a tile with key -1.  Returns the
// lane's place in the tile's list.
__device__ __forceinline__ int warp_tile_add(int* at, int key) {
    const int lane = threadIdx.x & 31;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const int leader = __ffs(peers) - 1;
    int base = 0;
    if (key >= 0 && lane == leader) base = atomicAdd(&at[key], __popc(peers));
    return __shfl_sync(0xffffffffu, base, leader) + __popc(peers & ((1u << lane) - 1u));
}

// Per-marker preparation: contact cell, arc length ds (min-image,
// immersed_boundary.cpp:164-173), stencil origin, validity, and the tile
// occupancy counts.  Also starts the step's counters and per-channel
// results at zero (nothing else of the step runs before it, and the previous
// step's have been read): as memsets these were five graph nodes in a row.
// One thread per marker, or (QUAD, by interp_by_quads) four: a column and a
// row of the stencil each, one of the two neighbours' distances, and every
// fourth tile, as in k_tile_fill.  Both and the slots between them: 720 markers
// 28.5 -> 24.4 us, 72,000 37.8 -> 43.7, 204,528 52.6 -> 73.2.
template <typename R, bool QUAD>
__global__ void k_marker_prep(const ChannelDev* __restrict__ chans, int nch,
                              const CapsuleDev* __restrict__ caps, int M, MarkerBufs mb,
                              const double* __restrict__ phi_tbl, TileBufs tb, ContactBufs cb,
                              unsigned* status) {
    chain_begin();
    constexpr int LANES = QUAD ? 4 : 1;
    const int t = blockIdx.x * blockDim.x + threadIdx.x, m = t / LANES, q = t % LANES;
    for (int c = t; c < nch; c += gridDim.x * blockDim.x) {
        tb.capped[c] = 0;
        tb.fluid_touched[c] = 0;
        tb.resid_gate[c] = 0u;
        tb.resid_plain[c] = 0u;
    }
    if (t < NUM_STEP_CTR) tb.ctr[t] = 0;
    const bool in = m < M;   // (lanes beyond the last marker only take part)
    const ChannelDev& ch = chans[in ? mb.mk_chan[m] : 0];
    const double2 p = in ? mb.pos[m] : make_double2(0.0, 0.0);
    if (in && q == LANES - 1 && !ch.brute_contact) {
        const int c = ch.cell_base + contact_cell(ch, p);
        cb.cell_of[m] = c;
        cb.next[m] = atomicExch(&cb.cell[c].x, m + 1);
    }
    double ds = 0.0;
    {
        double dp = 0.0, dn = 0.0;
        if (in) {
            const CapsuleDev& cp = caps[mb.mk_cap[m]];
            const int k = m - cp.off, n = cp.n;
            const int kp = cp.off + (k - 1 + n) % n, kn = cp.off + (k + 1) % n;
            const double Lx = (double)ch.nx;
            if constexpr (QUAD) {
                const double2 o = mb.pos[(q & 1) ? kn : kp];
                dp = norm_d((q & 1) ? min_image_d(o, p, Lx) : min_image_d(p, o, Lx));
            } else {
                dp = norm_d(min_image_d(p, mb.pos[kp], Lx));
                dn = norm_d(min_image_d(mb.pos[kn], p, Lx));
            }
        }
        if constexpr (QUAD) {
            dn = __shfl_sync(0xffffffffu, dp, 1, 4);
            dp = __shfl_sync(0xffffffffu, dp, 0, 4);
        }
        ds = 0.5 * (dp + dn);
    }
    bool ok = in && finite2(p);
    int ix0 = 0, iy0 = 0;
    if (ok) {
        // markers more than one period outside the lattice are skipped (the
        // reference indexes out of range there); wrapped x stays in [0, nx)
        if (p.x < -(double)ch.nx + 2.0 || p.x >= 2.0 * (double)ch.nx - 3.0) ok = false;
        if (fabs(p.y) > 1e9) ok = false;
        if (ok) {
            ix0 = (int)floor(p.x);
            iy0 = (int)floor(p.y);
            if (iy0 < -2 || iy0 >= ch.ny + 2) ok = false;
        }
    } else if (in && q == 0) {
        atomicOr(status, (unsigned)ST_NAN_MARKER);
    }
    if (in && q == 0) {
        mb.org[m] = make_int2(ix0, iy0);
        mb.valid[m] = ok;
    }
    // Peskin weights of the stencil, evaluated once per step (delta_function.h:44-59)
    double wx[4], wy[4];
    if constexpr (QUAD) {
        const double ax = ok ? phi_lut(phi_tbl, p.x - (double)(ix0 - 1 + q)) : 0.0;
        wy[0] = ok ? phi_lut(phi_tbl, p.y - (double)(iy0 - 1 + q)) : 0.0;   // this lane's row
#pragma unroll
        for (int k = 0; k < 4; ++k) wx[k] = __shfl_sync(0xffffffffu, ax, k, 4);
        if (ok) {
            if constexpr (sizeof(R) == 8) {
                if (q == 0) mb.ds[m] = ds;
                mb.wx[t] = ax;
                mb.wy[t] = wy[0];
            } else {
                if (q == 0) mb.dsf[m] = (float)ds;
                reinterpret_cast<float*>(mb.wxf)[t] = (float)ax;
                reinterpret_cast<float*>(mb.wyf)[t] = (float)wy[0];
            }
        }
    } else if (ok) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            wx[k] = phi_lut(phi_tbl, p.x - (double)(ix0 - 1 + k));
            wy[k] = phi_lut(phi_tbl, p.y - (double)(iy0 - 1 + k));
        }
        if constexpr (sizeof(R) == 8) {
            mb.ds[m] = ds;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                mb.wx[4 * (size_t)m + k] = wx[k];
                mb.wy[4 * (size_t)m + k] = wy[k];
            }
        } else {
            mb.dsf[m] = (float)ds;
            mb.wxf[m] = make_float4((float)wx[0], (float)wx[1], (float)wx[2], (float)wx[3]);
            mb.wyf[m] = make_float4((float)wy[0], (float)wy[1], (float)wy[2], (float)wy[3]);
        }
    }
    if constexpr (sizeof(R) == 4) {
        if (ok) {
            auto point = [&](int k, int j) {
                const double w = wx[k] * wy[j];
                return w > 1e-15 ? (float)w : (w > 0.5e-15 ? WF_TOUCH_ONLY : WF_NONE);
            };
#pragma unroll
            for (int j = 0; j < 4 / LANES; ++j)   // (QUAD: the lane's own row)
                mb.wf[4 * (size_t)m + q + j] =
                    make_float4(point(0, j), point(1, j), point(2, j), point(3, j));
        }
    }
    int tiles[8];
    const int nt = ok ? stencil_tiles(ch, ix0, iy0, tiles) : 0;
#pragma unroll
    for (int a = 0; a < 8; a += LANES) {
        int key = -1;
#pragma unroll
        for (int l = 0; l < LANES; ++l)
            if (l == q && a + l < nt) key = tiles[a + l];
        // (most stencils lie in one or two tiles)
        if (__any_sync(0xffffffffu, key >= 0)) warp_tile_add(tb.tile_cnt, key);
    }
}

// Slot map of the step, and per slot the record the spread reads first
// (SlotInfo: tile, channel, tile origin, list length and offset, nx, ny), so
// that a spread warp starts a slot with one 32-byte load.  One thread per
// tile: a warp takes slots and list space for its touched tiles with one
// atomic each (which numbers they get does not matter to any result), so no
// scan runs before it.  The tile's count is cleared for the next step and
// tile_pos[t] is left at the tile's first list entry for k_tile_fill.
// Each slot is also entered under its list-length class (slot_order), for the
// spread's work order.  The blocks after the tiles' build the contact cells.
__global__ void k_tile_slots(const ChannelDev* __restrict__ chans, int M, MarkerBufs mb,
                             TileBufs tb, int* tile_slot, ContactBufs cb,
                             int tile_blocks) {
    chain_begin();
    if ((int)blockIdx.x >= tile_blocks) {
        contact_cells((blockIdx.x - tile_blocks) * blockDim.x + threadIdx.x, M, chans, mb, cb,
                      &tb.ctr[CTR_CONTACT]);
        return;
    }
    const int t = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    const int cnt = t < tb.T ? tb.tile_cnt[t] : 0;
    const unsigned touched = __ballot_sync(0xffffffffu, cnt > 0);
    if (touched == 0u) {                       // warp-uniform
        if (t < tb.T) tile_slot[t] = -1;
        return;
    }
    int inc = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    int sbase = 0, lbase = 0;
    if (lane == 31) {
        sbase = atomicAdd(&tb.ctr[CTR_SLOTS], __popc(touched));
        lbase = atomicAdd(&tb.ctr[CTR_LIST], inc);
    }
    sbase = __shfl_sync(0xffffffffu, sbase, 31);
    lbase = __shfl_sync(0xffffffffu, lbase, 31);
    if (cnt > 0) {
        const int s = sbase + __popc(touched & ((1u << lane) - 1u)), off = lbase + inc - cnt;
        tb.tile_cnt[t] = 0;
        tb.tile_pos[t] = off;
        tile_slot[t] = s;
        const int chan = tb.tile_chan[t];
        const ChannelDev& ch = chans[chan];
        const int local = t - ch.tile_base;
        SlotInfo si;
        si.tile = t;
        si.chan = chan;
        si.x0 = (local % ch.tiles_x) * TILE_W;
        si.y0 = (local / ch.tiles_x) * TILE_H;
        si.cnt = cnt;
        si.off = off;
        si.nx = ch.nx;
        si.ny = ch.ny;
        tb.slot_info[s] = si;
        // rank within the list-length class: one atomic per class and warp
        const int cls = slot_class(cnt);
        const unsigned peers = __match_any_sync(__activemask(), cls);
        const int leader = __ffs(peers) - 1;
        int base = 0;
        if (lane == leader) base = atomicAdd(&tb.ctr[CTR_CLASS + cls], __popc(peers));
        base = __shfl_sync(peers, base, leader);
        tb.slot_order[(size_t)cls * tb.max_slots + base + __popc(peers & ((1u << lane) - 1u))] = s;
    } else if (t < tb.T) {
        tile_slot[t] = -1;
    }
}

// The spread's work order: slots by descending class, any order within a
// class (every slot's result is independent of the warp and of the order).
// Lane l holds the first position of class SLOT_CLASSES - 1 - l, so a
// position's class is the last lane whose start does not exceed it.
struct WorkOrder {
    int start;
    __device__ __forceinline__ explicit WorkOrder(const int* __restrict__ ctr) {
        const int lane = threadIdx.x & 31;
        const int n = lane < SLOT_CLASSES ? ctr[CTR_CLASS + SLOT_CLASSES - 1 - lane] : 0;
        int inc = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        start = inc - n;
    }
    // (all lanes of the warp call it with the same position)
    __device__ __forceinline__ int slot(const int* __restrict__ order, int max_slots, int p) const {
        const bool below = (threadIdx.x & 31) < SLOT_CLASSES && start <= p;
        const int l = __popc(__ballot_sync(0xffffffffu, below)) - 1;
        const int s0 = __shfl_sync(0xffffffffu, start, l);
        return order[(size_t)(SLOT_CLASSES - 1 - l) * max_slots + p - s0];
    }
};

template <bool QUAD>
__global__ void k_tile_fill(const ChannelDev* __restrict__ chans, int M, MarkerBufs mb,
                            int* tile_pos, int* __restrict__ list, const int* tile_slot) {
    chain_begin();
    constexpr int LANES = QUAD ? 4 : 1;
    const int t = blockIdx.x * blockDim.x + threadIdx.x, m = t / LANES, q = t % LANES;
    const bool ok = m < M && mb.valid[m];   // (the others only take part)
    const ChannelDev& ch = chans[ok ? mb.mk_chan[m] : 0];
    const int2 og = ok ? mb.org[m] : make_int2(0, 0);
    // the lanes of a tile take consecutive list entries (an FP64 spread
    // restores the order)
    int tiles[8];
    const int nt = ok ? stencil_tiles(ch, og.x, og.y, tiles) : 0;
#pragma unroll
    for (int a = 0; a < 8; a += LANES) {
        int key = -1;
#pragma unroll
        for (int l = 0; l < LANES; ++l)
            if (l == q && a + l < nt) key = tiles[a + l];
        if (__any_sync(0xffffffffu, key >= 0)) {
            const int at = warp_tile_add(tile_pos, key);
            if (key >= 0) list[at] = m;
        }
    }
    // the slot of every stencil cell, by row tile and stencil column, for the
    // interpolations of the step (one 32-byte record instead of 16 lookups)
    if (ok) {
        const int ty0 = first_tile_row(og.y, ch.ny), ty1 = last_tile_row(og.y, ch.ny);
        int s8[8];
#pragma unroll
        for (int sx = 0; sx < 4; ++sx) {
            if (QUAD && sx != q) continue;
            int jx = og.x - 1 + sx;
            if (jx < 0) jx += ch.nx;
            if (jx >= ch.nx) jx -= ch.nx;
            const bool in = jx >= 0 && jx < ch.nx;
            const int tx = in ? jx / TILE_W : 0;
            s8[sx] = in ? tile_slot[ch.tile_base + ty0 * ch.tiles_x + tx] : -1;
            s8[4 + sx] = in ? tile_slot[ch.tile_base + ty1 * ch.tiles_x + tx] : -1;
            if constexpr (QUAD) {
                mb.slot8[8 * (size_t)m + sx] = s8[sx];
                mb.slot8[8 * (size_t)m + 4 + sx] = s8[4 + sx];
            }
        }
        if constexpr (!QUAD) {
            int4* o = reinterpret_cast<int4*>(mb.slot8 + 8 * (size_t)m);
            o[0] = make_int4(s8[0], s8[1], s8[2], s8[3]);
            o[1] = make_int4(s8[4], s8[5], s8[6], s8[7]);
        }
    }
}

constexpr int SPREAD_WARPS = 8;       // force tiles processed per CTA (one per warp)
constexpr int SPREAD_LIST_MAX = 4096; // longer lists are clamped and flagged

// The tile accumulators keep rows of TILE_W + 4 cells: the 4 x 4 stencil
// points of a marker (4 consecutive rows and columns) then fall on 16
// distinct banks (a row stride of 32 puts all 4 rows on the same banks).
constexpr int ACC_W = TILE_W + 4;
constexpr int ACC_CELLS = TILE_H * ACC_W;
__device__ __forceinline__ int acc_at(int c) { return (c / TILE_W) * ACC_W + (c % TILE_W); }

// Deterministic spread into force tiles for MDF sweep `sweep` (FP64 contexts, bit
// for bit; the FP32-arithmetic modes run k_spread_fx).  Sweep 0 spreads the
// membrane + contact forces (immersed_boundary.cpp:25-100); sweep k >= 1 adds the
// corrections dF (:231-286).  A warp owns a tile, or (WIDE) a band of eight of its
// columns, a CTA of four warps the tile (spread_wide.cuh): either way every cell
// receives its contributions in the reference's order.  On a channel's last sweep the
// warps also add the body force on FLUID cells, apply the force cap and count capped
// cells (simulation.cpp:540-609), writing the final tile force `fin`.  Tiles are dealt
// to the warps or CTAs in rounds over the work order (longest lists first, alternating
// direction, so that each share sums to about the same work; a shared
// claim counter serialises on one L2 address); the next tile's record is fetched
// while the current one is processed.
//
// Few tiles leave the chip idle, and a tile's chain is then the kernel's length, which
// four warps cut; with many tiles the bands' passes over each list are only more work.
// The line lies where the warps with a tile each (24 an SM) run in one round and the
// bands' CTAs (6 an SM) in three.  It goes by the tiles touched when the context is
// initialized, as large lattices with few markers have many tiles too.  Spread
// phase of a step of five sweeps, a warp a tile / bands, us, by touched tiles:
//   200 to 800 x 40 to 160 channels    103   73  55     1161 100  76     2528 125 114
//                                     4985  142 185     9055 224 294    17342 372 546
//   lattices of 1024 x 256 and more    132   96  62      832  99  83     1664 115 116
//                                     2128  156 136     3264 158 192     4128 188 226
//   four capsules of 300 nodes          15  206 148 (lists of up to 300)
constexpr int BAND_TILES = 2800;
template <bool WIDE> using SpreadTile = typename std::conditional<WIDE, BandTile, WarpTile>::type;
template <bool WIDE> constexpr int spread_warps = WIDE ? BAND_WARPS : SPREAD_WARPS;
template <bool WIDE>
constexpr size_t spread_smem =
    sizeof(SpreadTile<WIDE>) * spread_warps<WIDE> + (WIDE ? sizeof(int) * SORT_SMEM : 0);

template <bool WIDE>
__global__ void __launch_bounds__(32 * spread_warps<WIDE>, WIDE ? 6 : 3)
k_spread(const ChannelDev* __restrict__ chans, const SlotInfo* __restrict__ slot_info,
         const int* __restrict__ slot_order, const int* __restrict__ ctr, int max_slots,
         int* __restrict__ list, MarkerBufs mb, double* __restrict__ acc,
         double* __restrict__ acc0, double* __restrict__ gsnap, double* __restrict__ fin,
         int sweep, int mode, const unsigned* __restrict__ resid_gate,
         const int* __restrict__ plain_needed, int* __restrict__ capped,
         int* __restrict__ fluid_touched, unsigned* status) {
    if (sweep > 0 && mode == MDF_PLAIN && plain_needed && !*plain_needed) return;
    using Tile = SpreadTile<WIDE>;
    constexpr int THREADS = WIDE ? 32 * BAND_WARPS : 32;   // of the group that has a tile
    extern __shared__ __align__(16) unsigned char spread_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    Tile& B = reinterpret_cast<Tile*>(spread_raw)[warp];
    int* sort = WIDE ? reinterpret_cast<int*>(reinterpret_cast<Tile*>(spread_raw) + BAND_WARPS)
                     : reinterpret_cast<int*>(B.v);
    const int group = WIDE ? blockIdx.x : blockIdx.x * SPREAD_WARPS + warp;
    const int groups = WIDE ? gridDim.x : gridDim.x * SPREAD_WARPS;
    const int gt = WIDE ? threadIdx.x : lane;
    const int n_slots = ctr[CTR_SLOTS];
    const WorkOrder wo(ctr);
    int round = 0, next = group;
    int nslot = next < n_slots ? wo.slot(slot_order, max_slots, next) : 0;
    SlotInfo nfo{};
    if (next < n_slots) nfo = slot_info[nslot];
    while (next < n_slots) {   // uniform in the group
        const int slot = nslot;
        const SlotInfo si = nfo;
        ++round;
        next = round * groups + ((round & 1) ? groups - 1 - group : group);
        if (next < n_slots) {
            nslot = wo.slot(slot_order, max_slots, next);
            nfo = slot_info[nslot];
        }
        const int chan = si.chan;
        const ChannelDev& ch = chans[chan];
        const int K = ch.ibm_iterations > 1 ? ch.ibm_iterations : 1;
        if (sweep >= K) continue;
        if (sweep > 0 && !mdf_active(ch, mode, resid_gate, chan)) continue;  // sweep 0: all
        int cnt = si.cnt;
        if (cnt > SPREAD_LIST_MAX) {
            if (gt == 0) atomicOr(status, (unsigned)ST_LIST_OVERFLOW);
            cnt = SPREAD_LIST_MAX;
        }
        int* lst = list + si.off;
        const int first = sweep == 0
                              ? tile_list_sort<THREADS>(lst, cnt, sort, gt, !WIDE || K > 1)
                              : (lane < cnt ? lst[lane] : 0);
        const bool last = mode == MDF_LEARNED ? true : (mode == MDF_SEED ? false : sweep == K - 1);
        // a learned channel's membrane-only force lives in acc0 only: the
        // seed sweep and a fallback's restart read it there.  The
        // accumulators hold (x, y) pairs per cell: [slot][TILE_CELLS] double2.
        const double2* src = reinterpret_cast<const double2*>(
            (ch.learned && (mode == MDF_SEED || (mode == MDF_PLAIN && sweep == 1))) ? acc0 : acc);
        const size_t base = (size_t)slot * 2 * TILE_CELLS, base2 = (size_t)slot * TILE_CELLS;
        // this lane's cells: column a, rows b and b + 4 of the band, or a column of
        // the tile
        constexpr int MINE = WIDE ? 2 : TILE_H;
        const int mine_x = WIDE ? BAND_W * warp + (lane & 7) : lane;
        auto row_of = [&](int h) { return WIDE ? (lane >> 3) + 4 * h : h; };
        auto at = [&](int r) { return r * Tile::ROW + (WIDE ? lane & 7 : lane); };
        __syncwarp();
#pragma unroll
        for (int h = 0; h < MINE; ++h) {
            const int r = row_of(h), c = r * TILE_W + mine_x;
            const double2 a = sweep > 0 ? src[base2 + c] : make_double2(0.0, 0.0);
            B.ax[at(r)] = a.x;
            B.ay[at(r)] = a.y;
            if (last && K > 1) {
                gsnap[base + c] = a.x;
                gsnap[base + TILE_CELLS + c] = a.y;
            }
        }
        const double2* frc = sweep == 0 ? mb.frc : mb.dF;
        auto org_of = [&](int m) { return mb.org[m]; };
        auto load = [&](int m, int sy, BandMarker& k) {
            k.f = frc[m];
            k.org = mb.org[m];
            k.ds = mb.ds[m];
            const double2* wx2 = reinterpret_cast<const double2*>(mb.wx + 4 * (size_t)m);
            const double2 wa = wx2[0], wb = wx2[1];
            k.wx[0] = wa.x; k.wx[1] = wa.y; k.wx[2] = wb.x; k.wx[3] = wb.y;
            k.wy = mb.wy[4 * (size_t)m + sy];
        };
        if constexpr (WIDE) {
            band_spread<true>(B, lst, cnt, first, si.nx, si.ny, si.x0 + BAND_W * warp, 0, si.y0,
                              lane, org_of, load);
        } else if (si.nx > TILE_W) {
            band_spread<false>(B, lst, cnt, first, si.nx, si.ny, si.x0, 0, si.y0, lane, org_of,
                               load);
        } else {
            for (int col = 0; col < TILE_W; col += BAND_W)
                band_spread<true>(B, lst, cnt, first, si.nx, si.ny, si.x0 + col, col, si.y0, lane,
                                  org_of, load);
        }
        if (!last) {
            double2* out = reinterpret_cast<double2*>((sweep == 0 && ch.learned) ? acc0 : acc);
#pragma unroll
            for (int h = 0; h < MINE; ++h) {
                const int r = row_of(h);
                out[base2 + r * TILE_W + mine_x] = make_double2(B.ax[at(r)], B.ay[at(r)]);
            }
            continue;
        }
        // finalize: body force on FLUID cells, then the force cap
        int n_cap = 0, n_fluid = 0;
        const double Fm = ch.max_force, Fm2 = Fm * Fm;
        const bool body = (ch.body_fx != 0.0 || ch.body_fy != 0.0);
#pragma unroll
        for (int h = 0; h < MINE; ++h) {
            const int r = row_of(h), c = r * TILE_W + mine_x;
            const int jx = si.x0 + mine_x, jy = si.y0 + r;
            double vx = B.ax[at(r)], vy = B.ay[at(r)];
            if (jx < si.nx && jy < si.ny) {
                const bool fluid = cell_kind(ch, jx, jy) == CK_FLUID;
                if (fluid && body) {
                    vx += ch.body_fx;
                    vy += ch.body_fy;
                }
                const double f2 = vx * vx + vy * vy;
                if (f2 > Fm2) {
                    const double sc = Fm / sqrt(f2);
                    vx *= sc;
                    vy *= sc;
                    ++n_cap;
                }
                n_fluid += fluid ? 1 : 0;
            }
            // (no sweep reads acc after a channel's last one)
            fin[base + c] = vx;
            fin[base + TILE_CELLS + c] = vy;
        }
        n_cap = __reduce_add_sync(0xffffffffu, n_cap);
        n_fluid = __reduce_add_sync(0xffffffffu, n_fluid);
        if (lane == 0) {
            if (n_cap) atomicAdd(&capped[chan], n_cap);
            if (n_fluid) atomicAdd(&fluid_touched[chan], n_fluid);
        }
    }
}

// The spread of the FP32-arithmetic modes (FP32 and FP16-shifted storage):
// the reference's contributions (f w) ds of each stencil point with
// w > 1e-15, formed as (float)f (float)w (float)ds and summed per cell
// exactly in fixed point.  Integer addition does not depend on the order of the
// terms, so the lanes of a warp add any markers' points in any order, with
// 32-bit shared-memory atomics, and the result is the same on every run, in
// every launch shape and whether a channel runs alone or in an ensemble; the
// marker lists need no sort.  Each value is v = q 2^-38 with the integer q
// split into a low part of 20 bits (unsigned, in [0, 2^20)) and a high part
// (signed).  A cell takes at most one term per list entry (channels at
// least 4 cells wide), so at most SPREAD_LIST_MAX = 4,096 low parts a sweep,
// whose sum stays below 2^32; the high parts are summed modulo 2^32, exact
// while the cell's sum stays below 2^13 in magnitude, far beyond any
// lattice force.
//
// A cell that no stencil point of the tile's markers reaches (with weight
// above 1e-15) receives nothing in any sweep of the step (the lists do not
// change between sweeps) and so holds zero throughout; about five in six
// cells of a tile are such.  The accumulators are therefore read and written
// only at the touched cells: a sweep adds its sum, rounded to float once, to
// the previous sweep's value there, and the readers of the accumulators (the
// interpolations, at the same stencil points) read nothing else.  The last
// sweep writes every cell of the tile's final force and of the force before
// that sweep, zero plus the body force where untouched.  The shared
// accumulators start at zero once per kernel and are cleared again at the
// touched cells after each tile.  FP64 contexts keep k_spread (the
// reference's serial order, bit for bit).
constexpr int FX_LO_BITS = 20;
constexpr float FX_SCALE = 274877906944.0f;          // 2^38
constexpr float FX_UNSCALE = 1.0f / 274877906944.0f;  // 2^-38 (exact)
struct SpreadFxWarp {
    unsigned lo[2][ACC_CELLS];        // x, y; rows of ACC_W cells
    int hi[2][ACC_CELLS];
    unsigned char hit[ACC_CELLS];     // touched this tile
    unsigned short idx[TILE_CELLS];   // the touched cells, compacted
};
// A tile is one warp's work, eight tiles a CTA, or (WIDE) a CTA's of four warps.
// Where the tiles are few, the sweep takes as long as one tile's chain of marker
// passes and cells, which four warps cut by four; where they are many, the
// narrow form keeps more tiles in flight, and its waits cost less.  The line goes by
// the slots a context may need, its lattice tiles or 8 a marker, of contexts with
// capsules all over; a large lattice with few markers stays with one warp, which was
// its only form before (4096 x 1024 with 10 capsules, five sweeps, 134 us a step).
// Spread phase of a step of five sweeps, one warp / two / four / eight a tile, us, by
// lattice tiles:
//   400 x 80, 130 tiles                  66.4  53.1  44.9  44.4
//   12 ragged channels, about 1,000      76.3  54.8  50.1  49.6
//   16 channels of 512 x 104, 3,300      83.7  57.4  53.1  56.3
//   32 channels, 6,600                   93.0  67.3  75.9  82.0
//   64 channels, 13,000                  98.1  99.8 105.3 120.4
//   4096 x 1024, 16,384 (one sweep)      20.3        29.0
constexpr int FX_WIDE_WARPS = 4, FX_WIDE_SLOTS = 8192;
template <bool WIDE> constexpr int fx_threads = 32 * (WIDE ? FX_WIDE_WARPS : SPREAD_WARPS);
template <bool WIDE> constexpr size_t fx_smem = sizeof(SpreadFxWarp) * (WIDE ? 1 : SPREAD_WARPS);
__device__ __forceinline__ long long fx_quant(float v) { return __float2ll_rn(v * FX_SCALE); }
__device__ __forceinline__ unsigned fx_lo(long long q) {
    return (unsigned)(q & ((1LL << FX_LO_BITS) - 1));
}
__device__ __forceinline__ int fx_hi(long long q) { return (int)(q >> FX_LO_BITS); }
__device__ __forceinline__ float fx_value(unsigned lo, int hi) {
    return __ll2float_rn((long long)hi * (1LL << FX_LO_BITS) + (long long)lo) * FX_UNSCALE;
}

template <bool WIDE>
__global__ void __launch_bounds__(fx_threads<WIDE>, WIDE ? 8 : 4)
k_spread_fx(const ChannelDev* __restrict__ chans, const SlotInfo* __restrict__ slot_info,
            const int* __restrict__ slot_order, const int* __restrict__ ctr, int max_slots,
            const int* __restrict__ list, MarkerBufs mb,
            double* __restrict__ acc, double* __restrict__ acc0, float* __restrict__ gsnap,
            float* __restrict__ fin, int sweep, int mode, const unsigned* __restrict__ resid_gate,
            const int* __restrict__ plain_needed, int* __restrict__ capped,
            int* __restrict__ fluid_touched, unsigned* status) {
    if (sweep > 0 && mode == MDF_PLAIN && plain_needed && !*plain_needed) return;
    extern __shared__ __align__(16) unsigned char spread_fx_raw[];
    // the group of WPT warps that works on a tile, its warp `wg` and thread `gl`
    constexpr int WPT = WIDE ? FX_WIDE_WARPS : 1, GROUPS = fx_threads<WIDE> / (32 * WPT);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int group = warp / WPT, wg = warp % WPT, gl = 32 * wg + lane;
    auto group_sync = [] {
        if constexpr (WIDE) __syncthreads(); else __syncwarp();
    };
    SpreadFxWarp& W = reinterpret_cast<SpreadFxWarp*>(spread_fx_raw)[group];
    for (int i = gl; i < ACC_CELLS; i += 32 * WPT) {
        W.lo[0][i] = W.lo[1][i] = 0u;
        W.hi[0][i] = W.hi[1][i] = 0;
        W.hit[i] = 0;
    }
    group_sync();
    const int n_slots = ctr[CTR_SLOTS];
    const WorkOrder wo(ctr);
    const int ngroups = gridDim.x * GROUPS;
    // round k takes work-order positions k ngroups .. (k + 1) ngroups - 1,
    // the groups in reverse order on odd rounds
    const int wid = blockIdx.x * GROUPS + group;
    int round = 0, next = wid;
    int nslot = next < n_slots ? wo.slot(slot_order, max_slots, next) : 0;
    SlotInfo nfo{};
    if (next < n_slots) nfo = slot_info[nslot];
    while (next < n_slots) {
        const int slot = nslot;
        const SlotInfo si = nfo;
        ++round;
        next = round * ngroups + ((round & 1) ? ngroups - 1 - wid : wid);
        if (next < n_slots) {
            nslot = wo.slot(slot_order, max_slots, next);
            nfo = slot_info[nslot];
        }
        const int chan = si.chan;
        const ChannelDev& ch = chans[chan];
        const int K = ch.ibm_iterations > 1 ? ch.ibm_iterations : 1;
        if (sweep >= K) continue;  // uniform in the group
        if (sweep > 0 && !mdf_active(ch, mode, resid_gate, chan)) continue;  // sweep 0: all
        const int nx = si.nx, ny = si.ny;
        const int x0 = si.x0, y0 = si.y0;
        int cnt = si.cnt;
        if (cnt > SPREAD_LIST_MAX) {
            if (gl == 0) atomicOr(status, (unsigned)ST_LIST_OVERFLOW);
            cnt = SPREAD_LIST_MAX;
        }
        const int* lst = list + si.off;
        const size_t base = (size_t)slot * 2 * TILE_CELLS;
        const bool last = mode == MDF_LEARNED ? true : (mode == MDF_SEED ? false : sweep == K - 1);
        // a learned channel's membrane-only force lives in acc0 only (k_spread)
        const float2* src = reinterpret_cast<const float2*>(
            (ch.learned && (mode == MDF_SEED || (mode == MDF_PLAIN && sweep == 1))) ? acc0 : acc);
        const size_t base2 = (size_t)slot * TILE_CELLS;
        // four lanes per marker, one stencil row each, eight markers a warp and pass;
        // the next pass's marker data is loaded before this pass's points.
        // Neighbouring list entries are neighbouring markers, whose stencils
        // overlap: the lanes of marker jm take their four columns in an order
        // rotated by jm, so that the warp's adds of one instruction meet
        // fewer of each other's cells (same-address shared atomics serialise;
        // along a vertical piece of membrane all eight markers share their
        // columns)
        const int jm = gl >> 2, sy = gl & 3;
        const bool rot1 = jm & 1, rot2 = jm & 2;
        struct Mk {
            float4 w;
            double2 f;
            float ds;
            int2 org;
        };
        auto fetch = [&](int c, Mk& k) {
            if (c + jm < cnt) {
                const int m = lst[c + jm];
                k.f = sweep == 0 ? mb.frc[m] : mb.dF[m];
                k.org = mb.org[m];
                k.ds = mb.dsf[m];
                k.w = mb.wf[4 * (size_t)m + sy];
            }
        };
        Mk cur{}, nxt{};
        fetch(0, cur);
        for (int c0 = 0; c0 < cnt; c0 += 8 * WPT) {
            fetch(c0 + 8 * WPT, nxt);
            const int iy = cur.org.y - 1 + sy, cyl = iy - y0;
            if (c0 + jm < cnt && cyl >= 0 && cyl < TILE_H && iy >= 0 && iy < ny) {
                const bool ok = !(isnan(cur.f.x) || isnan(cur.f.y));
                const float fx = (float)cur.f.x, fy = (float)cur.f.y, ds = cur.ds;
                const float4 a = rot1 ? make_float4(cur.w.y, cur.w.z, cur.w.w, cur.w.x) : cur.w;
                const float wr[4] = {rot2 ? a.z : a.x, rot2 ? a.w : a.y, rot2 ? a.x : a.z,
                                     rot2 ? a.y : a.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    int jx = cur.org.x - 1 + ((k + jm) & 3);
                    if (jx < 0) jx += nx;
                    if (jx >= nx) jx -= nx;
                    const int cl = jx - x0;
                    const float wf = wr[k];
                    // touched: a superset of the points that the
                    // interpolations read (they test the weight in float)
                    if (jx >= 0 && jx < nx && cl >= 0 && cl < TILE_W && wf != WF_NONE) {
                        const int i = cyl * ACC_W + cl;
                        W.hit[i] = 1;   // (lanes that meet here all store 1)
                        if (ok && wf != WF_TOUCH_ONLY) {
                            const long long qx = fx_quant(fx * wf * ds), qy = fx_quant(fy * wf * ds);
                            atomicAdd(&W.lo[0][i], fx_lo(qx));
                            atomicAdd(&W.hi[0][i], fx_hi(qx));
                            atomicAdd(&W.lo[1][i], fx_lo(qy));
                            atomicAdd(&W.hi[1][i], fx_hi(qy));
                        }
                    }
                }
            }
            cur = nxt;
        }
        group_sync();
        if (!last) {
            // the touched cells of the warp's rows, compacted row by row
            unsigned short* idx = W.idx + wg * (TILE_CELLS / WPT);
            int n = 0;
#pragma unroll
            for (int rr = 0; rr < TILE_H / WPT; ++rr) {
                const int r = wg * (TILE_H / WPT) + rr;
                const bool h = W.hit[r * ACC_W + lane] != 0;
                const unsigned b = __ballot_sync(0xffffffffu, h);
                if (h) idx[n + __popc(b & ((1u << lane) - 1u))] = (unsigned short)(r * TILE_W + lane);
                n += __popc(b);
            }
            __syncwarp();
            float2* out = reinterpret_cast<float2*>((sweep == 0 && ch.learned) ? acc0 : acc);
            for (int k = lane; k < n; k += 32) {
                const int c = idx[k], i = acc_at(c);
                float2 v = make_float2(fx_value(W.lo[0][i], W.hi[0][i]),
                                       fx_value(W.lo[1][i], W.hi[1][i]));
                if (sweep > 0) {
                    const float2 a = src[base2 + c];
                    v.x = a.x + v.x;
                    v.y = a.y + v.y;
                }
                out[base2 + c] = v;
                W.lo[0][i] = W.lo[1][i] = 0u;
                W.hi[0][i] = W.hi[1][i] = 0;
                W.hit[i] = 0;
            }
            group_sync();
            continue;
        }
        // finalize every cell, two adjacent cells a lane: the value before
        // this sweep (zero where untouched) plus this sweep's sum, the body
        // force on FLUID cells, then the force cap with the capped-cell
        // count (as k_spread, in float).  Cell kinds follow from the row
        // alone unless the channel has a cell-type mask or x boundaries.
        int n_cap = 0, n_fluid = 0;
        const float Fm = (float)ch.max_force, Fm2 = Fm * Fm;
        const float bfx = (float)ch.body_fx, bfy = (float)ch.body_fy;
        const bool body = (ch.body_fx != 0.0 || ch.body_fy != 0.0);
        const bool row_kinds = ch.mask == nullptr && ch.bc_x != 0 && ch.bc_x != 2;
        const float2 zero = make_float2(0.f, 0.f);
#pragma unroll 2
        for (int it = wg; it < TILE_H / 2; it += WPT) {
            const int r = 2 * it + (lane >> 4), cx = 2 * (lane & 15);
            const int c = r * TILE_W + cx, i = r * ACC_W + cx;
            const int jx = x0 + cx, jy = y0 + r;
            const bool h0 = W.hit[i] != 0, h1 = W.hit[i + 1] != 0;
            float2 a0 = zero, a1 = zero, v0 = zero, v1 = zero;
            if (h0 || h1) {
                if (sweep > 0) {
                    const float4 a = *reinterpret_cast<const float4*>(src + base2 + c);
                    if (h0) a0 = make_float2(a.x, a.y);
                    if (h1) a1 = make_float2(a.z, a.w);
                }
                if (h0) {
                    v0 = make_float2(a0.x + fx_value(W.lo[0][i], W.hi[0][i]),
                                     a0.y + fx_value(W.lo[1][i], W.hi[1][i]));
                    W.lo[0][i] = W.lo[1][i] = 0u;
                    W.hi[0][i] = W.hi[1][i] = 0;
                    W.hit[i] = 0;
                }
                if (h1) {
                    v1 = make_float2(a1.x + fx_value(W.lo[0][i + 1], W.hi[0][i + 1]),
                                     a1.y + fx_value(W.lo[1][i + 1], W.hi[1][i + 1]));
                    W.lo[0][i + 1] = W.lo[1][i + 1] = 0u;
                    W.hi[0][i + 1] = W.hi[1][i + 1] = 0;
                    W.hit[i + 1] = 0;
                }
            }
            if (K > 1) {
                *reinterpret_cast<float2*>(gsnap + base + c) = make_float2(a0.x, a1.x);
                *reinterpret_cast<float2*>(gsnap + base + TILE_CELLS + c) = make_float2(a0.y, a1.y);
            }
            float2 v[2] = {v0, v1};
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                if (jx + e < nx && jy < ny) {
                    const bool fluid =
                        row_kinds ? (ch.periodic_y || (jy != 0 && jy != ny - 1))
                                  : cell_kind(ch, jx + e, jy) == CK_FLUID;
                    if (fluid && body) {
                        v[e].x += bfx;
                        v[e].y += bfy;
                    }
                    const float f2 = v[e].x * v[e].x + v[e].y * v[e].y;
                    if (f2 > Fm2) {
                        const float sc = Fm / sqrtf(f2);
                        v[e].x *= sc;
                        v[e].y *= sc;
                        ++n_cap;
                    }
                    n_fluid += fluid ? 1 : 0;
                }
            }
            *reinterpret_cast<float2*>(fin + base + c) = make_float2(v[0].x, v[1].x);
            *reinterpret_cast<float2*>(fin + base + TILE_CELLS + c) = make_float2(v[0].y, v[1].y);
        }
        for (int o = 16; o > 0; o >>= 1) {
            n_cap += __shfl_down_sync(0xffffffffu, n_cap, o);
            n_fluid += __shfl_down_sync(0xffffffffu, n_fluid, o);
        }
        if (lane == 0) {
            if (n_cap) atomicAdd(&capped[chan], n_cap);
            if (n_fluid) atomicAdd(&fluid_touched[chan], n_fluid);
        }
        group_sync();
    }
}

// MDF correction of one sweep (immersed_boundary.cpp:231-286): interpolate
// u = (j + F/2)/rho with the force spread so far, then
// dF = 2 rho(nearest node) (U_prev - U_interp).  Also keeps the step's total
// correction (dFsum), the first sweep's interpolation (u0) and the no-slip
// residual max |U_prev - U_interp| per channel: at the learned form's sweep
// (resid_gate) and at a plain iteration's last sweep (resid_plain).
template <typename R, bool QUAD>
__global__ void k_mdf_interp(const ChannelDev* __restrict__ chans, int M, MarkerBufs mb,
                             const typename Mom4<R>::T* __restrict__ mom,
                             const double* __restrict__ acc, const double* __restrict__ acc0,
                             int sweep, int mode, unsigned* __restrict__ resid_gate,
                             unsigned* __restrict__ resid_plain,
                             const int* __restrict__ plain_needed) {
    if (mode == MDF_PLAIN && plain_needed && !*plain_needed) return;  // no channel needs it
    const int t = blockIdx.x * blockDim.x + threadIdx.x, m = QUAD ? t >> 2 : t;
    const int chan = m < M ? mb.mk_chan[m] : 0;
    const ChannelDev& ch = chans[chan];
    const bool on = m < M && sweep < ch.ibm_iterations && mb.valid[m] &&
                    mdf_active(ch, mode, resid_gate, chan);
    const double* base = (mode == MDF_PLAIN && ch.learned && sweep == 1) ? acc0 : acc;
    double rho_local;
    double2 u;
    if constexpr (QUAD) {
        u = quad_interp<R>(ch, mb, m, on, t & 3, mom, base, rho_local);
        if (!on || (t & 3) != 0) return;
    } else {
        if (!on) return;
        u = interp_u_mom<R, true>(ch, mb, m, mom, base, rho_local);
    }
    const double2 v = mb.vel[m];
    const double dux = v.x - u.x, duy = v.y - u.y;
    const double2 d = make_double2(dux * (2.0 * rho_local), duy * (2.0 * rho_local));
    mb.dF[m] = d;
    if (mode == MDF_PLAIN && sweep == 1) {
        mb.u0[m] = u;
        mb.dFsum[m] = d;
    } else {
        const double2 s0 = mb.dFsum[m];
        mb.dFsum[m] = make_double2(s0.x + d.x, s0.y + d.y);
    }
    // the per-channel residual max, one atomic per channel and warp
    const bool want = mode == MDF_LEARNED || sweep == ch.ibm_iterations - 1;
    warp_max_resid(mode == MDF_LEARNED ? resid_gate : resid_plain, chan, want,
                   sqrt(dux * dux + duy * duy));
}

// Whether any channel needs the plain correction sweeps this step: a forcing
// channel that is not learned, or a learned one whose gate residual is above
// its threshold.  One CTA; runs after the learned sweep's interpolation.
__global__ void k_plain_needed(const ChannelDev* __restrict__ chans, int nch,
                               const unsigned* __restrict__ resid_gate, int* __restrict__ flag) {
    __shared__ int any;
    if (threadIdx.x == 0) any = 0;
    __syncthreads();
    int mine = 0;
    for (int c = threadIdx.x; c < nch; c += blockDim.x) {
        const ChannelDev& ch = chans[c];
        if (ch.cap_end > ch.cap_begin && ch.ibm_iterations > 1 &&
            (!ch.learned || mdf_fallback(resid_gate[c], ch.mdf_threshold)))
            mine = 1;
    }
    if (mine) any = 1;
    __syncthreads();
    if (threadIdx.x == 0) *flag = any;
}

void launch_plain_needed(const ChannelDev* chans, int nch, TileBufs& tb, cudaStream_t st) {
    k_plain_needed<<<1, 256, 0, st>>>(chans, nch, tb.resid_gate, tb.plain_needed);
}

// (rho, jx, jy) of every cell of the step's force tiles, one warp per tile
// (rows of 32 cells: coalesced population loads).
template <typename S, typename R>
__global__ void k_tile_moments(const ChannelDev* __restrict__ chans,
                               const SlotInfo* __restrict__ slot_info,
                               const int* __restrict__ n_slots_p, const S* __restrict__ f,
                               typename Mom4<R>::T* __restrict__ mom) {
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const int n_slots = *n_slots_p;
    for (int slot = warp; slot < n_slots; slot += nwarps) {
        const SlotInfo si = slot_info[slot];
        const ChannelDev& ch = chans[si.chan];
        const int x0 = si.x0, y0 = si.y0;
        const int jx = x0 + lane;
        // four rows at a time: their 36 population loads are issued together
#pragma unroll
        for (int rb = 0; rb < TILE_H; rb += 4) {
            R v[4][9];
            bool use[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int jy = y0 + rb + i;
                use[i] = jx < ch.nx && jy < ch.ny && cell_kind(ch, jx, jy) != CK_SOLID;
                if (use[i]) {
                    const long long n = (long long)jy * ch.pitch + jx;
#pragma unroll
                    for (int q = 0; q < 9; ++q)
                        v[i][q] = PopIO<S, R>::ld(f + ch.f_off + q * ch.plane + n, q);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                typename Mom4<R>::T q;
                q.x = 0; q.y = 0; q.z = 0; q.w = 0;
                if (use[i]) {   // the cell's moments, in the working precision
                    R r, a, b;
                    lattice_moments(v[i], r, a, b);
                    q.x = (R)(double)r;
                    q.y = (R)(double)a;
                    q.z = (R)(double)b;
                }
                mom[(size_t)slot * TILE_CELLS + (rb + i) * TILE_W + lane] = q;
            }
        }
    }
}

// Moves marker m with its interpolated velocity u (simulation.cpp:656-675,
// capsule.cpp:267-297) and empties the record of its contact cell for the next
// step (every marker of a cell stores the same zeros).
__device__ __forceinline__ void move_marker(const ChannelDev& ch, const MarkerBufs& mb,
                                            const ContactBufs& cb, int m, double2 u) {
    if (!ch.brute_contact) cb.cell[cb.cell_of[m]] = make_int2(0, 0);
    double2 p = mb.pos[m];
    const double ux = u.x, uy = u.y;
    mb.vel[m] = make_double2(ux, uy);
    // the step's correction before its last sweep (the network's label, or
    // on a learned step its seed) becomes the next step's network input
    mb.dFprev[m] = (mb.valid[m] && ch.ibm_iterations > 1)
                       ? make_double2(mb.dFsum[m].x - mb.dF[m].x, mb.dFsum[m].y - mb.dF[m].y)
                       : make_double2(0.0, 0.0);
    p.x = p.x + ux * ch.dt;
    p.y = p.y + uy * ch.dt;
    const double Lx = (double)ch.nx;
    if (isfinite(p.x)) {
        // the reference wraps with while-loops (capsule.cpp:287-296); moves
        // are far below one period, so a bounded loop gives the same result
        int it = 0;
        while (p.x < 0.0 && it < 8) { p.x += Lx; ++it; }
        while (p.x >= Lx && it < 16) { p.x -= Lx; ++it; }
        if (p.x < 0.0 || p.x >= Lx) {
            p.x = fmod(p.x, Lx);
            if (p.x < 0.0) p.x += Lx;
        }
    }
    if (!ch.periodic_y) {
        const double ymin = 1.5, ymax = (double)ch.ny - 1.5;
        if (p.y < ymin) p.y = ymin;
        if (p.y > ymax) p.y = ymax;
    }
    mb.pos[m] = p;
}

// Interpolate the new velocity and move the markers (FP64 contexts), one
// thread per marker or (QUAD) four, by interp_by_quads: 2400 markers 14.7 us a
// launch with one thread, 6.7 with four (divisions and 144 loads in a row).
template <bool QUAD>
__global__ void k_interp_move(const ChannelDev* __restrict__ chans, int M, MarkerBufs mb,
                              ContactBufs cb, const double* __restrict__ f,
                              const double* __restrict__ fin) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, m = QUAD ? t >> 2 : t;
    if constexpr (QUAD) {
        const ChannelDev& ch = chans[m < M ? mb.mk_chan[m] : 0];
        const double2 u = quad_interp_acc(ch, mb, m, m < M && mb.valid[m], t & 3, f, fin);
        if (m < M && (t & 3) == 0) move_marker(ch, mb, cb, m, u);
    } else {
        if (m >= M) return;
        const ChannelDev& ch = chans[mb.mk_chan[m]];
        double2 u = make_double2(0.0, 0.0);
        if (mb.valid[m]) u = interp_u_acc(ch, mb, m, f, fin);
        move_marker(ch, mb, cb, m, u);
    }
}

// The marker move of the FP32-arithmetic modes, one block per capsule: the
// block first forms, for every cell of the box that holds the capsule's
// stencils, the new state's velocity (0 on SOLID cells) from its moments and
// the cell's final force, into shared memory, the threads running along the
// box's rows (each cell's nine populations are read once, coalesced, where
// the markers' stencils overlap, and divided once); then one thread per
// marker interpolates from there with the terms, order and arithmetic of
// interp_u_acc (the same values, so the same result bit for bit), and moves
// it.  A capsule whose box exceeds MOVE_BOX_MAX cells interpolates from global
// memory as k_interp_move does.
//
// Bound: latency, of few capsules as of many (each thread's loads depend on the
// marker's cell, then on the cell's tile); so all of a cell's loads are issued at
// once and few registers are held, and the block is as wide as the capsule has
// cells (100-130 of 24 markers) where all blocks are resident at once, half of
// that where they are not and every warp's own forming of the box counts.  One
// warp per capsule, with five floats a cell in shared memory and 126 registers,
// then blocks of 128 threads, of 64 and of 32 (us):
//   30 capsules, FP32         13.5   9.4  10.3
//   40 capsules, FP16S        21.0  11.1  12.6
//   2000 capsules, FP32       33.4  23.3  22.5  27.9
//   8522 capsules, FP16S      68.0  54.9  44.3  41.7

// The new state's velocity of a cell, jy in [0, ny).
template <typename S>
__device__ __forceinline__ float2 new_velocity(const ChannelDev& ch, int jx, int jy,
                                               const S* __restrict__ f,
                                               const int* __restrict__ tile_slot,
                                               const float* __restrict__ fin) {
    const long long nn = (long long)jy * ch.pitch + jx;
    float v[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) v[q] = PopIO<S, float>::ld(f + ch.f_off + q * ch.plane + nn, q);
    const int sl = tile_slot[ch.tile_base + (jy / TILE_H) * ch.tiles_x + jx / TILE_W];
    if (cell_kind(ch, jx, jy) == CK_SOLID) return make_float2(0.f, 0.f);
    float gx = 0.f, gy = 0.f, rho, a, b;
    if (sl >= 0) {
        const int cell = (jy % TILE_H) * TILE_W + (jx % TILE_W);
        gx = fin[(size_t)sl * 2 * TILE_CELLS + cell];
        gy = fin[(size_t)sl * 2 * TILE_CELLS + TILE_CELLS + cell];
    }
    lattice_moments(v, rho, a, b);
    if (!(rho > 1e-15f)) return make_float2(0.f, 0.f);
    const float inv = __frcp_rn(rho);
    return make_float2((a + 0.5f * gx) * inv, (b + 0.5f * gy) * inv);
}

constexpr int MOVE_BOX_MAX = 512;
constexpr int MOVE_WIDE_CAPS = 1024;
template <typename S, int MOVE_THREADS>
__global__ void __launch_bounds__(MOVE_THREADS)
k_interp_move_caps(const CapsuleDev* __restrict__ caps, const ChannelDev* __restrict__ chans,
                   MarkerBufs mb, ContactBufs cb, const S* __restrict__ f,
                   const int* __restrict__ tile_slot, const float* __restrict__ fin) {
    __shared__ float2 uv[MOVE_BOX_MAX];
    const int tid = threadIdx.x, lane = tid & 31;
    const CapsuleDev cp = caps[blockIdx.x];
    const ChannelDev& ch = chans[cp.chan];
    const int nx = ch.nx, ny = ch.ny, n = cp.n, off = cp.off;
    // the stencils' box: x relative to the first valid marker (minimum
    // image); every warp forms it for itself
    int ref = 0, dmin = INT_MAX, dmax = INT_MIN, ymin = INT_MAX, ymax = INT_MIN;
    bool have = false;
    for (int k0 = 0; k0 < n; k0 += 32) {
        const int k = k0 + lane;
        const bool v = k < n && mb.valid[off + k];
        const int2 og = v ? mb.org[off + k] : make_int2(0, 0);
        const unsigned vm = __ballot_sync(0xffffffffu, v);
        if (!have && vm) {
            ref = __shfl_sync(0xffffffffu, og.x, __ffs(vm) - 1);
            have = true;
        }
        if (v) {
            int d = og.x - ref;
            if (2 * d > nx) d -= nx;
            if (2 * d < -nx) d += nx;
            dmin = min(dmin, d);
            dmax = max(dmax, d);
            ymin = min(ymin, og.y);
            ymax = max(ymax, og.y);
        }
    }
    dmin = __reduce_min_sync(0xffffffffu, dmin);
    dmax = __reduce_max_sync(0xffffffffu, dmax);
    ymin = __reduce_min_sync(0xffffffffu, ymin);
    ymax = __reduce_max_sync(0xffffffffu, ymax);
    const int bw = dmax - dmin + 4, bh = ymax - ymin + 4;
    const bool boxed = have && (long long)bw * bh <= MOVE_BOX_MAX;
    if (boxed) {
        const int bx0 = ref + dmin - 1, by0 = ymin - 1;
        for (int i = tid; i < bw * bh; i += MOVE_THREADS) {
            const int by = i / bw, bx = i - by * bw;
            int jx = (bx0 + bx) % nx;
            if (jx < 0) jx += nx;
            const int jy = by0 + by;
            float2 u = make_float2(0.f, 0.f);
            if (jy >= 0 && jy < ny) u = new_velocity(ch, jx, jy, f, tile_slot, fin);
            uv[i] = u;
        }
    }
    __syncthreads();
    for (int k = tid; k < n; k += MOVE_THREADS) {
        const int m = off + k;
        double2 u = make_double2(0.0, 0.0);
        if (mb.valid[m]) {
            const int ix0 = mb.org[m].x, iy0 = mb.org[m].y;
            float wxs[4], wys[4];
            stencil_weights(mb, m, wxs, wys);
            float ux = 0.f, uy = 0.f;
            if (boxed) {
                int d = ix0 - ref;
                if (2 * d > nx) d -= nx;
                if (2 * d < -nx) d += nx;
#pragma unroll
                for (int sy = 0; sy < 4; ++sy) {
                    const int jy = iy0 - 1 + sy;
                    if (jy < 0 || jy >= ny) continue;
                    const int row = (iy0 - ymin + sy) * bw + (d - dmin);
#pragma unroll
                    for (int sx = 0; sx < 4; ++sx) {
                        const float w = wxs[sx] * wys[sy];
                        if (w > 1e-15f) {
                            const float2 c = uv[row + sx];
                            ux += c.x * w;
                            uy += c.y * w;
                        }
                    }
                }
            } else {
#pragma unroll 1
                for (int tap = 0; tap < 16; ++tap) {
                    const int sy = tap >> 2, sx = tap & 3, jy = iy0 - 1 + sy;
                    const float wx = sx < 2 ? (sx ? wxs[1] : wxs[0]) : (sx == 2 ? wxs[2] : wxs[3]);
                    const float wy = sy < 2 ? (sy ? wys[1] : wys[0]) : (sy == 2 ? wys[2] : wys[3]);
                    const float w = wx * wy;
                    if (jy < 0 || jy >= ny || !(w > 1e-15f)) continue;
                    int jx = (ix0 - 1 + sx) % nx;
                    if (jx < 0) jx += nx;
                    const float2 c = new_velocity(ch, jx, jy, f, tile_slot, fin);
                    ux += c.x * w;
                    uy += c.y * w;
                }
            }
            u = make_double2((double)ux, (double)uy);
        }
        move_marker(ch, mb, cb, m, u);
    }
}

// ============================ launch wrappers ==============================

size_t membrane_smem_bytes(int maxn) {
    return (size_t)MEM_WARPS * MEM_DOUBLES_PER_NODE * maxn * sizeof(double);
}

bool spread_wide(bool fp64, int max_slots, int touched) {
    return fp64 ? touched <= BAND_TILES : max_slots <= FX_WIDE_SLOTS;
}

int spread_blocks_per_sm(bool fp64, bool wide) {
    int b = 0;
    const cudaError_t e =
        fp64 && wide ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                           &b, k_spread<true>, 32 * spread_warps<true>, spread_smem<true>)
        : fp64 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                     &b, k_spread<false>, 32 * spread_warps<false>, spread_smem<false>)
        : wide ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_spread_fx<true>,
                                                               fx_threads<true>, fx_smem<true>)
               : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_spread_fx<false>,
                                                               fx_threads<false>, fx_smem<false>);
    if (e != cudaSuccess || b < 1) b = 1;
    return b;
}

cudaError_t prepare_spread() {
    const cudaError_t e =
        cudaFuncSetAttribute(k_spread_fx<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)fx_smem<false>);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_spread<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)spread_smem<false>);
}

// ---------------- capsule geometry (thermo) ---------------------------------
// One thread per capsule, FP64 in the reference's serial order:
// Capsule::centroid, area, perimeter, secondMoments, deformationIndex and
// inclinationAngle (capsule.cpp:159-266).  Unwrapped nodes are regenerated
// on the fly (p_0 = X_0, p_i = p_{i-1} + minImage(X_i - X_{i-1})).
__device__ __forceinline__ double2 unwrap_next(const double2* X, int i, double2 p, double Lx) {
    const double2 d = min_image_d(X[i], X[i - 1], Lx);
    return make_double2(p.x + d.x, p.y + d.y);
}

__device__ void capsule_moments(const double2* X, int n, double Lx, double& mxx, double& myy,
                                double& mxy) {
    // capsule.cpp:209-247
    double A = 0.0, cx = 0.0, cy = 0.0;
    double2 a = X[0];
    const double2 p0 = a;
    for (int i = 0; i < n; ++i) {
        const double2 b = (i + 1 < n) ? unwrap_next(X, i + 1, a, Lx) : p0;
        const double cr = a.x * b.y - b.x * a.y;
        A += cr;
        cx += (a.x + b.x) * cr;
        cy += (a.y + b.y) * cr;
        a = b;
    }
    A *= 0.5;
    mxx = myy = mxy = 0.0;
    if (fabs(A) < 1e-15) return;
    cx /= (6.0 * A);
    cy /= (6.0 * A);
    a = p0;
    for (int i = 0; i < n; ++i) {
        const double2 q = (i + 1 < n) ? unwrap_next(X, i + 1, a, Lx) : p0;
        const double x0 = a.x - cx, y0 = a.y - cy;
        const double x1 = q.x - cx, y1 = q.y - cy;
        const double cr = x0 * y1 - x1 * y0;
        mxx += (x0 * x0 + x0 * x1 + x1 * x1) * cr;
        myy += (y0 * y0 + y0 * y1 + y1 * y1) * cr;
        mxy += (x0 * y1 + 2.0 * x0 * y0 + 2.0 * x1 * y1 + x1 * y0) * cr;
        a = q;
    }
    const double sgn = (A > 0.0) ? 1.0 : -1.0;
    mxx *= sgn / 12.0;
    myy *= sgn / 12.0;
    mxy *= sgn / 24.0;
}

__global__ void k_capsule_stats(const CapsuleDev* __restrict__ caps, int ncaps,
                                const double2* __restrict__ pos, double* __restrict__ out) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncaps) return;
    const CapsuleDev cd = caps[c];
    const double2* X = pos + cd.off;
    const int n = cd.n;
    const double Lx = (double)cd.periodic_nx;
    double* o = out + 6LL * c;
    // centroid (capsule.cpp:159-172)
    double2 cen = make_double2(0.0, 0.0);
    if (cd.periodic_nx > 0 && n > 0) {
        const double2 ref = X[0];
        double2 sum = ref;
        for (int i = 1; i < n; ++i) {
            const double2 d = min_image_d(X[i], ref, Lx);
            sum.x += ref.x + d.x;
            sum.y += ref.y + d.y;
        }
        cen = make_double2(sum.x / (double)n, sum.y / (double)n);
    } else if (n > 0) {
        for (int i = 0; i < n; ++i) {
            cen.x += X[i].x;
            cen.y += X[i].y;
        }
        cen = make_double2(cen.x / (double)n, cen.y / (double)n);
    }
    // area (capsule.cpp:174-195)
    double A = 0.0;
    if (cd.periodic_nx > 0 && n > 0) {
        double2 a = X[0];
        const double2 p0 = a;
        for (int i = 0; i < n; ++i) {
            const double2 b = (i + 1 < n) ? unwrap_next(X, i + 1, a, Lx) : p0;
            A += a.x * b.y - a.y * b.x;
            a = b;
        }
    } else {
        for (int i = 0; i < n; ++i) {
            const double2 a = X[i], b = X[(i + 1) % n];
            A += a.x * b.y - a.y * b.x;
        }
    }
    // perimeter (capsule.cpp:197-204)
    double P = 0.0;
    for (int i = 0; i < n; ++i) P += norm_d(min_image_d(X[(i + 1) % n], X[i], Lx));
    // deformation index and inclination (capsule.cpp:249-266)
    double D = 0.0, th = 0.0;
    if (n >= 3) {
        double mxx, myy, mxy;
        capsule_moments(X, n, Lx, mxx, myy, mxy);
        const double tr = 0.5 * (mxx + myy);
        const double dd = sqrt(0.25 * (mxx - myy) * (mxx - myy) + mxy * mxy);
        const double J1 = tr + dd;
        const double t2 = tr - dd;
        const double J2 = (t2 < 0.0) ? 0.0 : t2;
        const double s1 = sqrt(J1), s2 = sqrt(J2);
        D = (s1 + s2 > 1e-15) ? (s1 - s2) / (s1 + s2) : 0.0;
        th = 0.5 * atan2(2.0 * mxy, mxx - myy);
    }
    o[0] = cen.x;
    o[1] = cen.y;
    o[2] = 0.5 * fabs(A);
    o[3] = P;
    o[4] = D;
    o[5] = th;
}

void launch_capsule_stats(const CapsuleDev* caps, int ncaps, const double2* pos, double* out,
                          cudaStream_t st) {
    if (ncaps == 0) return;
    k_capsule_stats<<<(ncaps + 127) / 128, 128, 0, st>>>(caps, ncaps, pos, out);
}

cudaError_t prepare_membrane(int maxn) {
    const size_t smem = membrane_smem_bytes(maxn);
    if (smem <= 48 * 1024) return cudaSuccess;
    return cudaFuncSetAttribute(k_membrane, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)smem);
}

void launch_membrane(const CapsuleDev* caps, int ncaps, const MarkerBufs& mb, int* has_prev,
                     int maxn, unsigned* status, cudaStream_t st) {
    if (ncaps == 0) return;
    const size_t smem = membrane_smem_bytes(maxn);
    const int blocks = (ncaps + MEM_WARPS - 1) / MEM_WARPS;
    k_membrane<<<blocks, MEM_WARPS * 32, smem, st>>>(caps, ncaps, mb, has_prev, maxn, status);
}

// ---------------- obstacle repulsion (pillars) -------------------------------
// Obstacle::signedDistance / normalAt of CircleObstacle and RectObstacle
// (geometry/circle_obstacle.h:17-37, rect_obstacle.h:18-59) with the
// first-extremum semantics of std::min / std::max over initializer lists.
__device__ __forceinline__ double max3(double a, double b, double c) {
    double m = a;
    if (m < b) m = b;
    if (m < c) m = c;
    return m;
}
__device__ __forceinline__ double min4(double a, double b, double c, double d) {
    double m = a;
    if (b < m) m = b;
    if (c < m) m = c;
    if (d < m) m = d;
    return m;
}

__device__ void pillar_geometry(const double* o, double x, double y, double& sd, double2& nrm) {
    if (o[0] == 0.0) {   // circle (a, b) radius c
        const double dx = x - o[1], dy = y - o[2];
        const double d = sqrt(dx * dx + dy * dy);
        sd = d - o[3];
        nrm = (d < 1e-15) ? make_double2(1.0, 0.0) : make_double2(dx / d, dy / d);
        return;
    }
    const double x0 = o[1], y0 = o[2], x1 = o[3], y1 = o[4];
    {
        const double dx = max3(x0 - x, x - x1, 0.0);
        const double dy = max3(y0 - y, y - y1, 0.0);
        const double outside = sqrt(dx * dx + dy * dy);
        sd = (outside > 1e-15) ? outside : -min4(x - x0, x1 - x, y - y0, y1 - y);
    }
    // nearestPoint
    const double cx = (x < x0) ? x0 : ((x1 < x) ? x1 : x);
    const double cy = (y < y0) ? y0 : ((y1 < y) ? y1 : y);
    double2 np;
    if (cx == x && cy == y) {
        const double dl = x - x0, dr = x1 - x, db = y - y0, dt = y1 - y;
        const double dmin = min4(dl, dr, db, dt);
        if (dmin == dl) np = make_double2(x0, y);
        else if (dmin == dr) np = make_double2(x1, y);
        else if (dmin == db) np = make_double2(x, y0);
        else np = make_double2(x, y1);
    } else {
        np = make_double2(cx, cy);
    }
    const double ddx = x - np.x, ddy = y - np.y;
    const double d = sqrt(ddx * ddx + ddy * ddy);
    if (d < 1e-15) {
        const double dl = fabs(x - x0), dr = fabs(x - x1), db = fabs(y - y0), dt = fabs(y - y1);
        const double dmin = min4(dl, dr, db, dt);
        if (dmin == dl) nrm = make_double2(-1.0, 0.0);
        else if (dmin == dr) nrm = make_double2(1.0, 0.0);
        else if (dmin == db) nrm = make_double2(0.0, -1.0);
        else nrm = make_double2(0.0, 1.0);
    } else {
        nrm = make_double2(ddx / d, ddy / d);
    }
}

// RepulsionForce::computeObstacleRepulsion (repulsion.cpp:180-235) for every
// pillar of the marker's channel in order, after the pair contact.
__global__ void k_obstacle_repulsion(const ChannelDev* __restrict__ chans, int M, MarkerBufs mb) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    const ChannelDev& ch = chans[mb.mk_chan[m]];
    if (ch.n_pillars == 0) return;
    const double2 p = mb.pos[m], v = mb.vel[m];
    double2 f = mb.frc[m];
    const double r_cut = ch.rep_r_cut, eps = ch.rep_epsilon, sigma = ch.rep_sigma;
    const double gamma_n = ch.rep_damping, mu = ch.rep_friction;
    for (int k = 0; k < ch.n_pillars; ++k) {
        double sd;
        double2 nrm;
        pillar_geometry(ch.pillars + 5 * k, p.x, p.y, sd, nrm);
        if (sd >= r_cut) continue;
        double r = fabs(sd);
        if (r < 1e-15) r = 1e-15;
        const double F_rep = eps * pow(sigma / r, (double)ch.rep_power);
        if (sd < 0.0) {
            const double s = F_rep * 10.0;
            f.x += nrm.x * s;
            f.y += nrm.y * s;
            continue;
        }
        double F_n = F_rep;
        double2 F_t = make_double2(0.0, 0.0);
        if (gamma_n > 0.0 || mu > 0.0) {
            const double v_n = v.x * nrm.x + v.y * nrm.y;
            F_n = F_rep - gamma_n * v_n;
            if (F_n < 0.0) F_n = 0.0;
            if (mu > 0.0) {
                const double2 v_t = make_double2(v.x - nrm.x * v_n, v.y - nrm.y * v_n);
                const double v_t_mag = sqrt(v_t.x * v_t.x + v_t.y * v_t.y);
                if (v_t_mag > 1e-12) {
                    const double s = -mu * F_n;
                    F_t = make_double2((v_t.x / v_t_mag) * s, (v_t.y / v_t_mag) * s);
                }
            }
        }
        f.x += nrm.x * F_n + F_t.x;
        f.y += nrm.y * F_n + F_t.y;
    }
    mb.frc[m] = f;
}

void launch_obstacle_repulsion(const ChannelDev* chans, int M, const MarkerBufs& mb,
                               cudaStream_t st) {
    if (M == 0) return;
    k_obstacle_repulsion<<<(M + 255) / 256, 256, 0, st>>>(chans, M, mb);
}

void launch_contact_force(const ChannelDev* chans, int M, const MarkerBufs& mb,
                          const ContactBufs& cb, cudaStream_t st) {
    if (M == 0) return;
    const bool quads = interp_by_quads(M);
    const int B = 256, G = ((quads ? 4 * M : M) + B - 1) / B;
    (quads ? k_contact_force<true> : k_contact_force<false>)<<<G, B, 0, st>>>(chans, M, mb, cb);
}

template <typename R>
void launch_tiles(const ChannelDev* chans, int nch, const CapsuleDev* caps, int M,
                  const MarkerBufs& mb, TileBufs& tb, const ContactBufs& cb, int ncells, int parity,
                  const double* phi_tbl, unsigned* status, cudaStream_t st,
                  cudaEvent_t slots_ready) {
    const int B = 256, G = (M + B - 1) / B, TB = (tb.T + B - 1) / B;
    const bool quads = interp_by_quads(M);
    const int GM = ((quads ? 4 * M : M) + B - 1) / B;
    launch_chain(false, quads ? k_marker_prep<R, true> : k_marker_prep<R, false>, GM, B, 0, st,
                 chans, nch, caps, M, mb, phi_tbl, tb, cb, status);
    launch_chain(true, k_tile_slots, TB + (ncells > 0 ? G : 0), B, 0, st, chans, M, mb, tb,
                 tb.tile_slot[parity], cb, TB);
    if (slots_ready) cudaEventRecord(slots_ready, st);
    launch_chain(true, quads ? k_tile_fill<true> : k_tile_fill<false>, GM, B, 0, st, chans, M,
                 mb, tb.tile_pos, tb.list, tb.tile_slot[parity]);
}

template void launch_tiles<double>(const ChannelDev*, int, const CapsuleDev*, int, const MarkerBufs&,
                                   TileBufs&, const ContactBufs&, int, int, const double*,
                                   unsigned*, cudaStream_t, cudaEvent_t);
template void launch_tiles<float>(const ChannelDev*, int, const CapsuleDev*, int, const MarkerBufs&,
                                  TileBufs&, const ContactBufs&, int, int, const double*, unsigned*,
                                  cudaStream_t, cudaEvent_t);

template <typename R>
void launch_spread(const ChannelDev* chans, const MarkerBufs& mb, TileBufs& tb, int parity,
                   int sweep, int mode, int grid, unsigned* status, cudaStream_t st) {
    auto run = [&](auto kernel, int threads, size_t smem) {
        kernel<<<grid, threads, smem, st>>>(
            chans, tb.slot_info, tb.slot_order, tb.ctr, tb.max_slots, tb.list, mb, tb.acc, tb.acc0,
            static_cast<R*>(tb.gsnap), static_cast<R*>(tb.fin[parity]), sweep, mode, tb.resid_gate,
            tb.plain_needed, tb.capped, tb.fluid_touched, status);
    };
    if constexpr (sizeof(R) == 4) {
        if (tb.wide) run(k_spread_fx<true>, fx_threads<true>, fx_smem<true>);
        else run(k_spread_fx<false>, fx_threads<false>, fx_smem<false>);
    } else {
        if (tb.wide) run(k_spread<true>, 32 * spread_warps<true>, spread_smem<true>);
        else run(k_spread<false>, 32 * spread_warps<false>, spread_smem<false>);
    }
}
template void launch_spread<double>(const ChannelDev*, const MarkerBufs&, TileBufs&, int, int,
                                    int, int, unsigned*, cudaStream_t);
template void launch_spread<float>(const ChannelDev*, const MarkerBufs&, TileBufs&, int, int, int,
                                   int, unsigned*, cudaStream_t);

template <typename R>
void launch_mdf_interp(const ChannelDev* chans, int M, const MarkerBufs& mb, TileBufs& tb,
                       int sweep, int mode, cudaStream_t st) {
    const bool quads = interp_by_quads(M);
    const int B = tb.marker_block, G = ((quads ? 4 * M : M) + B - 1) / B;
    (quads ? k_mdf_interp<R, true> : k_mdf_interp<R, false>)<<<G, B, 0, st>>>(
        chans, M, mb, static_cast<const typename Mom4<R>::T*>(tb.mom), tb.acc, tb.acc0, sweep,
        mode, tb.resid_gate, tb.resid_plain, tb.plain_needed);
}
template void launch_mdf_interp<double>(const ChannelDev*, int, const MarkerBufs&, TileBufs&, int,
                                        int, cudaStream_t);
template void launch_mdf_interp<float>(const ChannelDev*, int, const MarkerBufs&, TileBufs&, int,
                                       int, cudaStream_t);

template <typename S, typename R>
void launch_tile_moments(const ChannelDev* chans, const S* f, TileBufs& tb, int grid,
                         cudaStream_t st) {
    k_tile_moments<S, R><<<grid, 256, 0, st>>>(chans, tb.slot_info, tb.ctr + CTR_SLOTS, f,
                                               static_cast<typename Mom4<R>::T*>(tb.mom));
}

template <typename S, typename R>
void launch_interp_move(const ChannelDev* chans, const CapsuleDev* caps, int ncaps, int M,
                        const MarkerBufs& mb, const ContactBufs& cb, const S* f, TileBufs& tb,
                        int parity, cudaStream_t st) {
    if constexpr (sizeof(R) == 4) {
        if (ncaps == 0) return;
        const float* fin = static_cast<const float*>(tb.fin[parity]);
        if (ncaps <= MOVE_WIDE_CAPS)
            k_interp_move_caps<S, 128><<<ncaps, 128, 0, st>>>(caps, chans, mb, cb, f,
                                                              tb.tile_slot[parity], fin);
        else
            k_interp_move_caps<S, 64><<<ncaps, 64, 0, st>>>(caps, chans, mb, cb, f,
                                                            tb.tile_slot[parity], fin);
    } else {
        const bool quads = interp_by_quads(M);
        const int B = tb.marker_block, G = ((quads ? 4 * M : M) + B - 1) / B;
        (quads ? k_interp_move<true> : k_interp_move<false>)<<<G, B, 0, st>>>(
            chans, M, mb, cb, f, static_cast<const double*>(tb.fin[parity]));
    }
}

#define SFG_INST(S, R)                                                                          \
    template void launch_tile_moments<S, R>(const ChannelDev*, const S*, TileBufs&, int,       \
                                            cudaStream_t);                                      \
    template void launch_interp_move<S, R>(const ChannelDev*, const CapsuleDev*, int, int,     \
                                           const MarkerBufs&, const ContactBufs&, const S*,    \
                                           TileBufs&, int, cudaStream_t);
SFG_INST(double, double)
SFG_INST(float, float)
SFG_INST(__half, float)
#undef SFG_INST

}  // namespace sfg

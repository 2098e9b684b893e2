// ibm_interp.cuh -- interpolation of the lattice velocity at a marker with
// the force accumulated so far, and the per-marker inputs of the learned
// multi-direct forcing network.  Shared by the plain forcing sweeps and the
// learned seed so that both interpolate identically.
#pragma once
#include <type_traits>
#include "markers.cuh"
#include "lattice.cuh"

namespace sfg {

// Slot of stencil cell (sx, jy) from the marker's slot record (k_tile_fill).
struct StencilSlots {
    int s[8];
    int ty0;
    __device__ __forceinline__ StencilSlots(const MarkerBufs& mb, int m, int iy0, int ny) {
        const int4* p = reinterpret_cast<const int4*>(mb.slot8 + 8 * (size_t)m);
        const int4 a = p[0], b = p[1];
        s[0] = a.x; s[1] = a.y; s[2] = a.z; s[3] = a.w;
        s[4] = b.x; s[5] = b.y; s[6] = b.z; s[7] = b.w;
        ty0 = first_tile_row(iy0, ny);
    }
    __device__ __forceinline__ int slot(int sx, int jy) const {
        return s[(jy / TILE_H != ty0 ? 4 : 0) + sx];
    }
};

// u = (j + F/2)/rho at the marker's 4 x 4 stencil with the final force acc
// (immersed_boundary.cpp:174-229 with the stencil weights of the step; SOLID rows and
// rho <= 1e-15 contribute zero).  FP64 contexts; the FP32-arithmetic modes move
// markers by capsule.
__device__ __forceinline__ double2 interp_u_acc(const ChannelDev& ch, const MarkerBufs& mb, int m,
                                               const double* __restrict__ f,
                                               const double* __restrict__ acc) {
    const int2 og = mb.org[m];
    const int ix0 = og.x, iy0 = og.y;
    const StencilSlots ss(mb, m, iy0, ch.ny);
    double wxs[4], wys[4];
    stencil_weights(mb, m, wxs, wys);
    int jxs[4];
#pragma unroll
    for (int sx = 0; sx < 4; ++sx) {
        int jx = ix0 - 1 + sx;
        if (jx < 0) jx += ch.nx;
        if (jx >= ch.nx) jx -= ch.nx;
        jxs[sx] = jx;
    }
    double ux = 0, uy = 0;
    // one stencil row at a time: the populations and forces of its four
    // cells are loaded together, then its terms are added in order
#pragma unroll
    for (int sy = 0; sy < 4; ++sy) {
        const int jy = iy0 - 1 + sy;
        double v[4][9], fx[4], fy[4];
        bool in[4], solid[4];
#pragma unroll
        for (int sx = 0; sx < 4; ++sx) {
            const int jx = jxs[sx];
            in[sx] = jy >= 0 && jy < ch.ny && jx >= 0 && jx < ch.nx;
            solid[sx] = in[sx] && cell_kind(ch, jx, jy) == CK_SOLID;
            if (in[sx] && !solid[sx]) {
                const long long n = (long long)jy * ch.pitch + jx;
#pragma unroll
                for (int q = 0; q < 9; ++q)
                    v[sx][q] = PopIO<double, double>::ld(f + ch.f_off + q * ch.plane + n, q);
                const size_t ci = (size_t)ss.slot(sx, jy) * 2 * TILE_CELLS +
                                  (jy % TILE_H) * TILE_W + (jx % TILE_W);
                fx[sx] = acc[ci];
                fy[sx] = acc[ci + TILE_CELLS];
            }
        }
#pragma unroll
        for (int sx = 0; sx < 4; ++sx) {
            if (!in[sx]) continue;
            const double w = wxs[sx] * wys[sy];
            if (w > 1e-15) {
                double rho = 0, jxm = 0, jym = 0, cu = 0, cv = 0;
                if (!solid[sx]) lattice_moments(v[sx], rho, jxm, jym);
                if (!solid[sx] && rho > 1e-15) {
                    cu = (jxm + 0.5 * fx[sx]) / rho;
                    cv = (jym + 0.5 * fy[sx]) / rho;
                }
                ux += cu * w;
                uy += cv * w;
            }
        }
    }
    return make_double2(ux, uy);
}

// Moments (rho, jx, jy) of a force tile's cells, computed once per step
// (k_tile_moments) because the populations do not change during the forcing
// sweeps: [slot][TILE_CELLS] records of R, rho = 0 on SOLID rows (where the
// reference's interpolation and density lookup give 0) and outside the
// channel.
template <typename R> struct Mom4;
template <> struct Mom4<double> { using T = double4; };
template <> struct Mom4<float> { using T = float4; };

// interp_u_acc with the step's tile moments and the accumulated force acc
// ([slot][TILE_CELLS] (x, y) pairs): the same terms in the same order.  The loads of
// a stencil row (moments and force of four cells) are issued together before any of
// their terms is formed, so a marker waits for one round of gathers per row instead of one per cell.  FP64
// divides by rho as the reference does (bit for bit); FP32-arithmetic modes
// multiply by one reciprocal per cell.  With NEAR, also the density
// at the node nearest to the marker (immersed_boundary.cpp:262-270: the
// node (int)(x + 0.5), (int)(y + 0.5), density 1 outside the lattice rows),
// taken from the stencil's moments already loaded (the node is stencil
// column and row 1 or 2).
template <typename R, bool NEAR = false>
__device__ __forceinline__ double2 interp_u_mom(const ChannelDev& ch, const MarkerBufs& mb, int m,
                                               const typename Mom4<R>::T* __restrict__ mom,
                                               const double* __restrict__ acc,
                                               double& rho_near) {
    // compute type: double in FP64 contexts (the reference's arithmetic),
    // float in the FP32-arithmetic modes (fewer registers, more resident
    // warps for this latency-bound gather)
    using C = typename std::conditional<sizeof(R) == 8, double, float>::type;
    const int2 og = mb.org[m];
    const int ix0 = og.x, iy0 = og.y;
    const StencilSlots ss(mb, m, iy0, ch.ny);
    C wxs[4], wys[4];
    stencil_weights(mb, m, wxs, wys);
    int jxs[4];
#pragma unroll
    for (int sx = 0; sx < 4; ++sx) {
        int jx = ix0 - 1 + sx;
        if (jx < 0) jx += ch.nx;
        if (jx >= ch.nx) jx -= ch.nx;
        jxs[sx] = jx;
    }
    // the nearest node's stencil column and row (-1: not wanted, or the
    // density is 1 outside the lattice rows)
    int sxn = -1, syn = -1;
    if (NEAR) {
        rho_near = 1.0;
        const double2 p = mb.pos[m];
        int ixr = (int)(p.x + 0.5);
        const int iyr = (int)(p.y + 0.5);
        if (ixr < 0) ixr += ch.nx;
        if (ixr >= ch.nx) ixr -= ch.nx;
        if (iyr >= 0 && iyr < ch.ny && ixr >= 0 && ixr < ch.nx) {
            sxn = (int)(p.x + 0.5) - ix0 + 1;
            syn = iyr - (iy0 - 1);
            // (always column and row 1 or 2 for a finite position; a
            // non-finite one keeps the density 1)
            if (sxn < 0 || sxn > 3 || syn < 0 || syn > 3) sxn = syn = -1;
        }
    }
    C ux = 0, uy = 0;
#pragma unroll
    for (int row = 0; row < 4; ++row) {
        typename Mom4<R>::T q[4];
        C fx[4], fy[4];
        bool in[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int sy = row, sx = i;
            const int jx = jxs[sx], jy = iy0 - 1 + sy;
            in[i] = jy >= 0 && jy < ch.ny && jx >= 0 && jx < ch.nx;
            const int sl = in[i] ? ss.slot(sx, jy) : -1;
            in[i] = in[i] && sl >= 0;
            if (in[i]) {
                const int cell = (jy % TILE_H) * TILE_W + (jx % TILE_W);
                q[i] = mom[(size_t)sl * TILE_CELLS + cell];
                // (x, y) pairs of R: double2 in FP64 contexts, float2 otherwise
                if constexpr (sizeof(R) == 8) {
                    const double2 a =
                        reinterpret_cast<const double2*>(acc)[(size_t)sl * TILE_CELLS + cell];
                    fx[i] = a.x;
                    fy[i] = a.y;
                } else {
                    const float2 a =
                        reinterpret_cast<const float2*>(acc)[(size_t)sl * TILE_CELLS + cell];
                    fx[i] = a.x;
                    fy[i] = a.y;
                }
            }
        }
        if (NEAR && row == syn) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (i == sxn && in[i]) rho_near = (double)q[i].x;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int sy = row, sx = i;
            if (!in[i]) continue;
            const C w = wxs[sx] * wys[sy];
            if (w > (C)1e-15) {
                const C rho = (C)q[i].x;
                C cu = 0, cv = 0;
                if (rho > (C)1e-15) {
                    if constexpr (sizeof(R) == 8) {
                        cu = ((double)q[i].y + 0.5 * fx[i]) / rho;
                        cv = ((double)q[i].z + 0.5 * fy[i]) / rho;
                    } else {
                        const float inv = __frcp_rn(rho);
                        cu = (q[i].y + 0.5f * fx[i]) * inv;
                        cv = (q[i].z + 0.5f * fy[i]) * inv;
                    }
                }
                ux += cu * w;
                uy += cv * w;
            }
        }
    }
    return make_double2((double)ux, (double)uy);
}

// interp_u_mom with four lanes per marker: lane `row` of the quad loads the four
// cells of its stencil row at once and forms their terms, then the rows' terms
// are added in the same order (row by row, the running sum passed from lane to
// lane), so the result is the one-thread sum bit for bit.  Every lane of the
// quad gets u and rho_near.  All lanes of the warp call this; a quad with
// on = false reads nothing.
template <typename R>
__device__ __forceinline__ double2 quad_interp(const ChannelDev& ch, const MarkerBufs& mb, int m,
                                               bool on, int row,
                                               const typename Mom4<R>::T* __restrict__ mom,
                                               const double* __restrict__ acc,
                                               double& rho_near) {
    // compute type: double in FP64 contexts (the reference's arithmetic),
    // float in the FP32-arithmetic modes
    using C = typename std::conditional<sizeof(R) == 8, double, float>::type;
    C tx[4], ty[4], near = 1;
    int syn = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) tx[i] = ty[i] = 0;
    if (on) {
        const int2 og = mb.org[m];
        const int jy = og.y - 1 + row;
        C wx[4], wy;
        int4 sl4;
        {
            const int ty0 = first_tile_row(og.y, ch.ny);
            sl4 = reinterpret_cast<const int4*>(mb.slot8 + 8 * (size_t)m)[jy / TILE_H != ty0 ? 1 : 0];
        }
        if constexpr (sizeof(R) == 8) {
            const double2* x2 = reinterpret_cast<const double2*>(mb.wx + 4 * (size_t)m);
            const double2 xa = x2[0], xb = x2[1];
            wx[0] = xa.x; wx[1] = xa.y; wx[2] = xb.x; wx[3] = xb.y;
            wy = mb.wy[4 * (size_t)m + row];
        } else {
            const float4 x = mb.wxf[m];
            wx[0] = x.x; wx[1] = x.y; wx[2] = x.z; wx[3] = x.w;
            wy = reinterpret_cast<const float*>(mb.wyf)[4 * (size_t)m + row];
        }
        const int sl[4] = {sl4.x, sl4.y, sl4.z, sl4.w};
        typename Mom4<R>::T q[4];
        C fx[4], fy[4];
        bool in[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            int jx = og.x - 1 + i;
            if (jx < 0) jx += ch.nx;
            if (jx >= ch.nx) jx -= ch.nx;
            in[i] = jy >= 0 && jy < ch.ny && jx >= 0 && jx < ch.nx && sl[i] >= 0;
            if (in[i]) {
                const size_t at = (size_t)sl[i] * TILE_CELLS + (jy % TILE_H) * TILE_W + (jx % TILE_W);
                q[i] = mom[at];
                // (x, y) pairs of R: double2 in FP64 contexts, float2 otherwise
                if constexpr (sizeof(R) == 8) {
                    const double2 a = reinterpret_cast<const double2*>(acc)[at];
                    fx[i] = a.x;
                    fy[i] = a.y;
                } else {
                    const float2 a = reinterpret_cast<const float2*>(acc)[at];
                    fx[i] = a.x;
                    fy[i] = a.y;
                }
            }
        }
        // the nearest node's stencil column and row (always 1 or 2 for a
        // finite position; otherwise, or outside the lattice, the density is 1)
        const double2 p = mb.pos[m];
        int ixr = (int)(p.x + 0.5);
        const int iyr = (int)(p.y + 0.5), sxn = ixr - og.x + 1;
        if (ixr < 0) ixr += ch.nx;
        if (ixr >= ch.nx) ixr -= ch.nx;
        syn = iyr - (og.y - 1);
        const bool seen = iyr >= 0 && iyr < ch.ny && ixr >= 0 && ixr < ch.nx && sxn >= 0 &&
                          sxn <= 3 && syn >= 0 && syn <= 3;
        syn = syn < 0 ? 0 : (syn > 3 ? 3 : syn);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (!in[i]) continue;
            if (seen && i == sxn) near = (C)q[i].x;
            const C w = wx[i] * wy;
            if (w > (C)1e-15) {
                const C rho = (C)q[i].x;
                C cu = 0, cv = 0;
                if (rho > (C)1e-15) {
                    if constexpr (sizeof(R) == 8) {
                        cu = ((double)q[i].y + 0.5 * fx[i]) / rho;
                        cv = ((double)q[i].z + 0.5 * fy[i]) / rho;
                    } else {
                        const float inv = __frcp_rn(rho);
                        cu = (q[i].y + 0.5f * fx[i]) * inv;
                        cv = (q[i].z + 0.5f * fy[i]) * inv;
                    }
                }
                tx[i] = cu * w;
                ty[i] = cv * w;
            }
        }
    }
    rho_near = (double)__shfl_sync(0xffffffffu, near, syn, 4);
    // a term that takes no part is +0, which leaves the sum as it is (it
    // starts at +0 and can never become -0)
    C ux = 0, uy = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const C sx = (((ux + tx[0]) + tx[1]) + tx[2]) + tx[3];
        const C sy = (((uy + ty[0]) + ty[1]) + ty[2]) + ty[3];
        ux = __shfl_sync(0xffffffffu, sx, r, 4);
        uy = __shfl_sync(0xffffffffu, sy, r, 4);
    }
    return make_double2((double)ux, (double)uy);
}

// interp_u_acc by four lanes of a warp, lane `row` a stencil row, as quad_interp.
__device__ __forceinline__ double2 quad_interp_acc(const ChannelDev& ch, const MarkerBufs& mb,
                                                   int m, bool on, int row,
                                                   const double* __restrict__ f,
                                                   const double* __restrict__ acc) {
    double tx[4], ty[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) tx[i] = ty[i] = 0;
    if (on) {
        const int2 og = mb.org[m];
        const int jy = og.y - 1 + row, ty0 = first_tile_row(og.y, ch.ny);
        const int4 sl4 =
            reinterpret_cast<const int4*>(mb.slot8 + 8 * (size_t)m)[jy / TILE_H != ty0 ? 1 : 0];
        const int sl[4] = {sl4.x, sl4.y, sl4.z, sl4.w};
        const double2* x2 = reinterpret_cast<const double2*>(mb.wx + 4 * (size_t)m);
        const double2 xa = x2[0], xb = x2[1];
        const double wx[4] = {xa.x, xa.y, xb.x, xb.y}, wy = mb.wy[4 * (size_t)m + row];
        double v[4][9], fx[4], fy[4];
        bool use[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            int jx = og.x - 1 + i;
            if (jx < 0) jx += ch.nx;
            if (jx >= ch.nx) jx -= ch.nx;
            use[i] = jy >= 0 && jy < ch.ny && jx >= 0 && jx < ch.nx &&
                     cell_kind(ch, jx, jy) != CK_SOLID;
            if (use[i]) {
                const long long n = (long long)jy * ch.pitch + jx;
#pragma unroll
                for (int q = 0; q < 9; ++q)
                    v[i][q] = PopIO<double, double>::ld(f + ch.f_off + q * ch.plane + n, q);
                const size_t ci =
                    (size_t)sl[i] * 2 * TILE_CELLS + (jy % TILE_H) * TILE_W + (jx % TILE_W);
                fx[i] = acc[ci];
                fy[i] = acc[ci + TILE_CELLS];
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const double w = wx[i] * wy;
            if (use[i] && w > 1e-15) {
                double rho, jxm, jym;
                lattice_moments(v[i], rho, jxm, jym);
                if (rho > 1e-15) {
                    tx[i] = (jxm + 0.5 * fx[i]) / rho * w;
                    ty[i] = (jym + 0.5 * fy[i]) / rho * w;
                }
            }
        }
    }
    double ux = 0, uy = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) {   // (see quad_interp)
        const double sx = (((ux + tx[0]) + tx[1]) + tx[2]) + tx[3];
        const double sy = (((uy + ty[0]) + ty[1]) + ty[2]) + ty[3];
        ux = __shfl_sync(0xffffffffu, sx, r, 4);
        uy = __shfl_sync(0xffffffffu, sy, r, 4);
    }
    return make_double2(ux, uy);
}

// Whether a per-marker kernel takes four lanes a marker.  Few markers
// cannot fill the chip and every kernel is one warp's chain of dependent loads
// and instructions, which the quad shortens (1,455 instructions a warp to a
// third; 720 markers: 8.6 -> 5.2 us a sweep); with many the one-thread form
// does the same loads with less work around them (204 k markers: the step's
// interpolations 111 us against 117).  The line lies where the quads' warps
// fill one resident wave of the chip.
inline bool interp_by_quads(int M) { return M <= 32768; }

// Inputs of the forcing network in the marker's local frame (tangent t along
// e_prev + e_next, normal n = (-t_y, t_x)):
//   [slip.t, slip.n, dF_prev.t, dF_prev.n, stretch, curvature, u_target.t,
//    u_target.n], slip = u_interp - u_target, u_target = the marker velocity
//   of the previous step (the forcing target, immersed_boundary.cpp:255),
//   stretch = (|e_prev| + |e_next|) / (L0_prev + L0_next) - 1,
//   curvature = atan2(e_prev x e_next, e_prev . e_next) / (0.5 (|e_prev| + |e_next|)).
__device__ __forceinline__ void mdf_features(const ChannelDev& ch, const CapsuleDev& cp,
                                             const MarkerBufs& mb, int m, double2 u_interp,
                                             float* feat, double2& t, double2& nrm) {
    const int k = m - cp.off, n = cp.n;
    const int kp = cp.off + (k - 1 + n) % n, kn = cp.off + (k + 1) % n;
    const double Lx = (double)ch.nx;
    const double2 p = mb.pos[m];
    const double2 ep = min_image_d(p, mb.pos[kp], Lx);
    const double2 en = min_image_d(mb.pos[kn], p, Lx);
    const double tx = ep.x + en.x, ty = ep.y + en.y;
    const double tl = sqrt(tx * tx + ty * ty);
    t = tl > 0.0 ? make_double2(tx / tl, ty / tl) : make_double2(1.0, 0.0);
    nrm = make_double2(-t.y, t.x);
    const double lp = norm_d(ep), ln = norm_d(en);
    const double stretch = (lp + ln) / (mb.rest_len[kp] + mb.rest_len[m]) - 1.0;
    const double curv = atan2(ep.x * en.y - ep.y * en.x, ep.x * en.x + ep.y * en.y) /
                        (0.5 * (lp + ln));
    const double2 ut = mb.vel[m];
    const double2 dp = mb.dFprev[m];
    const double sx = u_interp.x - ut.x, sy = u_interp.y - ut.y;
    feat[0] = (float)(sx * t.x + sy * t.y);
    feat[1] = (float)(sx * nrm.x + sy * nrm.y);
    feat[2] = (float)(dp.x * t.x + dp.y * t.y);
    feat[3] = (float)(dp.x * nrm.x + dp.y * nrm.y);
    feat[4] = (float)stretch;
    feat[5] = (float)curv;
    feat[6] = (float)(ut.x * t.x + ut.y * t.y);
    feat[7] = (float)(ut.x * nrm.x + ut.y * nrm.y);
}

// Per-channel maximum of a non-negative residual kept as float bits (NaN
// becomes the largest value, so it triggers the fallback).
__device__ __forceinline__ void atomic_max_resid(unsigned* slot, double r) {
    const float rf = (float)r;
    atomicMax(slot, isnan(rf) ? 0x7fc00000u : __float_as_uint(rf));
}

// atomic_max_resid for the active lanes of a warp (each calls it once, `on`
// lanes carry a residual; lanes that left the kernel take no part): lanes of
// one channel are reduced first and one lane per channel updates the slot (the max
// of non-negative floats is the max of their bit patterns, NaN mapped above every finite value as in atomic_max_resid).
__device__ __forceinline__ void warp_max_resid(unsigned* slots, int chan, bool on, double r) {
    const float rf = (float)r;
    const unsigned v = on ? (isnan(rf) ? 0x7fc00000u : __float_as_uint(rf)) : 0u;
    const unsigned key = on ? (unsigned)chan : 0xffffffffu;
    const unsigned peers = __match_any_sync(__activemask(), key);
    const unsigned m = __reduce_max_sync(peers, v);   // over the lanes of one key
    const int leader = __ffs(peers) - 1;
    if (on && (threadIdx.x & 31) == leader) atomicMax(&slots[chan], m);
}

}  // namespace sfg

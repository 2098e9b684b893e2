// markers.cuh -- Lagrangian-side kernels: membrane forces, soft contact,
// immersed-boundary force tiles, deterministic spreading, multi-direct
// forcing, and interpolate + move.
//
// All marker arithmetic is FP64 and is compiled without FMA contraction, so
// with the reference's evaluation order the results agree with the
// reference engine to the last bit wherever the same libm-class functions are
// not involved (atan2 in Helfrich bending and pow in the contact law are the
// exceptions, agreeing to a few ulp).
#pragma once
#include "common.cuh"

namespace sfg {

struct MarkerBufs {
    double2* pos;
    double2* vel;
    double2* frc;       // membrane + contact force (reference Capsule::forces_)
    double2* dF;        // MDF correction of the current sweep
    double* ds;         // arc length per marker (min-image)
    double* rest_len;
    double* rest_ang;
    double* rest_ds;
    double* prev_len;
    int* mk_cap;        // capsule of each marker
    int* mk_chan;       // channel of each marker
    int2* org;          // stencil origin of the step: floor(x), floor(y)
    int* valid;         // finite position with its stencil rows near the lattice
    int* pair_count;    // contact pairs visited per marker (bookkeeping)
    // Stencil weights of the step, phi(x - ix) for ix = ix0-1 .. ix0+2 and
    // phi(y - iy) for iy = iy0-1 .. iy0+2: in FP64 contexts the doubles; in the
    // FP32-arithmetic modes what their kernels compute with, formed once
    double* wx;         // [M][4] FP64 contexts
    double* wy;
    float4* wxf;        // [M] the weights rounded to float (interpolations)
    float4* wyf;
    float4* wf;         // [M][4] spread weight of each stencil row's points: the double
                        // product rounded to float, or one of the marks below
    float* dsf;         // [M] arc length rounded to float
    // multi-direct forcing state of the learned form and its training data
    double2* u0;        // velocity interpolated after the membrane-force spread
    double2* dFsum;     // forcing correction of this step summed over its sweeps
    double2* dFprev;    // previous step's correction before its last sweep
    // force-tile slots of the marker's stencil, this step: [M][2][4] =
    // [row tile (of the first / last stencil row)][stencil column sx]
    int* slot8;
};

// Marks in MarkerBufs::wf of points that take no part in the spread: a weight
// of at most 1e-15 that the interpolations may still read (they test a float
// product), and one that nothing reads.
constexpr float WF_TOUCH_ONLY = -1.0f;
constexpr float WF_NONE = -2.0f;

// The marker's stencil weights in the compute type of a context.
__device__ __forceinline__ void stencil_weights(const MarkerBufs& mb, int m, double wx[4],
                                                double wy[4]) {
    const double2* x2 = reinterpret_cast<const double2*>(mb.wx + 4 * (size_t)m);
    const double2* y2 = reinterpret_cast<const double2*>(mb.wy + 4 * (size_t)m);
    const double2 xa = x2[0], xb = x2[1], ya = y2[0], yb = y2[1];
    wx[0] = xa.x; wx[1] = xa.y; wx[2] = xb.x; wx[3] = xb.y;
    wy[0] = ya.x; wy[1] = ya.y; wy[2] = yb.x; wy[3] = yb.y;
}
__device__ __forceinline__ void stencil_weights(const MarkerBufs& mb, int m, float wx[4],
                                                float wy[4]) {
    const float4 x = mb.wxf[m], y = mb.wyf[m];
    wx[0] = x.x; wx[1] = x.y; wx[2] = x.z; wx[3] = x.w;
    wy[0] = y.x; wy[1] = y.y; wy[2] = y.z; wy[3] = y.w;
}

// ---------------- Peskin 4-point delta via the 1024-bin table --------------
// reference delta_function.h:44-54 (table built on the host from :18-26)
__device__ __forceinline__ double phi_lut(const double* tbl, double r) {
    double ar = fabs(r);
    if (ar >= 2.0) return 0.0;
    double idx = ar * (1024 * 0.5);
    int i = (int)idx;
    if (i >= 1024) return 0.0;
    double frac = idx - (double)i;
    return tbl[i] * (1.0 - frac) + tbl[i + 1] * frac;
}

__device__ __forceinline__ double2 min_image_d(double2 a, double2 b, double Lx) {
    double2 d = make_double2(a.x - b.x, a.y - b.y);
    if (Lx > 0.0) {
        if (d.x > 0.5 * Lx) d.x -= Lx;
        if (d.x < -0.5 * Lx) d.x += Lx;
    }
    return d;
}
__device__ __forceinline__ double norm_d(double2 a) { return sqrt(a.x * a.x + a.y * a.y); }

__device__ __forceinline__ bool finite2(double2 p) {
    return !(isnan(p.x) || isnan(p.y) || isinf(p.x) || isinf(p.y));
}

}  // namespace sfg

"""Division by the collision operators' constants through a reciprocal and two
fused multiply-adds: exactly the rounded quotient, and the cells that the method
does not cover (values near the ends of the exponent range, infinities, NaN) give
what division gives."""
from fractions import Fraction

import numpy as np
import pytest

CS2 = 1.0 / 3.0
CS4 = CS2 * CS2
CONSTANTS = [CS2, 2 * CS2, 2 * CS4, 9.0, 36.0, 18.0, 6.0, 12.0]


def _fma(a, b, c):
    """The correctly rounded a b + c (a Fraction converts to the nearest double);
    an exact zero takes the sign of the floating-point sum of the terms."""
    v = Fraction(a) * Fraction(b) + Fraction(c)
    return float(v) if v else a * b + c


def _div(a, d):
    y = 1.0 / d
    q0 = a * y
    return _fma(-_fma(d, q0, -a), y, q0)


def _hardest(d, count):
    """Dividends whose quotient lies nearest to the middle of two doubles: with
    integers D (53 bits, odd part) and an odd M (54 bits), a 2^k = M D + j with
    small j, so M = -j / D modulo 2^k."""
    num, den = Fraction(d).numerator, Fraction(d).denominator
    D = num if num > 1 else den
    while D % 2 == 0:
        D //= 2
    out = []
    for k in {max(D.bit_length() - 1, 1), D.bit_length(), 1, 2, 3}:
        inv = pow(D, -1, 1 << k)
        for j in range(1, count):
            for s in (-j, j):
                M0 = (s * inv) % (1 << k)
                for top in (1 << 53, (1 << 54) - (1 << k)):
                    M = top + M0 if top + M0 < 1 << 54 else M0 + (1 << 53)
                    v = (M * D - s) >> k
                    if 0 < v < 1 << 53 and M % 2:
                        out.append(float(v))
    return out


@pytest.mark.parametrize("d", CONSTANTS)
def test_reciprocal_is_good_enough(d):
    assert abs(Fraction(1.0 / d) * Fraction(d) - 1) <= Fraction(1, 1 << 54)


@pytest.mark.parametrize("d", CONSTANTS)
def test_quotient_is_correctly_rounded(d):
    rng = np.random.default_rng(5)
    m = rng.integers(1 << 52, 1 << 53, 4000).astype(float)
    a = np.concatenate([m, m[:500] * 2.0 ** rng.integers(-900, 900, 500),
                        np.arange(1.0, 300.0), (2.0 ** 53) - np.arange(1.0, 200.0)])
    hard = _hardest(d, 300)
    assert len(hard) > 50
    for v in [*a.tolist(), *hard]:
        for w in (v, -v):
            assert _div(w, d) == w / d


@pytest.mark.parametrize("d", CONSTANTS)
def test_sign_of_zero_is_kept(d):
    for z in (0.0, -0.0):
        assert np.signbit(_div(z, d)) == np.signbit(z / d)


# ------------------------------------------------------------------ on the GPU

CX = np.array([0, 1, 0, -1, 0, 1, -1, -1, 1.0])
CY = np.array([0, 0, 1, 0, -1, 1, 1, -1, -1.0])
W = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4)


def _velocity(f):
    rho = f[0] + f[1] + f[2] + f[3] + f[4] + f[5] + f[6] + f[7] + f[8]
    jx = f[1] - f[3] + f[5] - f[6] - f[7] + f[8]
    jy = f[2] - f[4] + f[5] + f[6] - f[7] - f[8]
    if rho > 1e-15:
        return rho, jx / rho, jy / rho
    return rho, np.float64(0), np.float64(0)


def _regularized(f, omega):
    rho, ux, uy = _velocity(f)
    fe = []
    for q in range(9):
        eu = CX[q] * ux + CY[q] * uy
        uu = ux * ux + uy * uy
        fe.append(W[q] * rho * (1 + eu / CS2 + (eu * eu) / (2 * CS4) - uu / (2 * CS2)))
    jx = jy = pxx = pxy = pyy = np.float64(0)
    for q in range(9):
        n = f[q] - fe[q]
        jx = jx + n * CX[q]
        jy = jy + n * CY[q]
        pxx = pxx + n * CX[q] * CX[q]
        pxy = pxy + n * CX[q] * CY[q]
        pyy = pyy + n * CY[q] * CY[q]
    out = []
    for q in range(9):
        qxx, qxy, qyy = CX[q] * CX[q] - CS2, CX[q] * CY[q], CY[q] * CY[q] - CS2
        reg = W[q] * ((CX[q] * jx + CY[q] * jy) / CS2 +
                      (qxx * pxx + 2.0 * qxy * pxy + qyy * pyy) / (2.0 * CS2 * CS2))
        out.append(fe[q] + (1 - omega) * reg + 0.0)
    return np.array(out)


@pytest.mark.gpu
@pytest.mark.parametrize("nx", [64, 63])
@pytest.mark.parametrize("kind", ["plain", "small", "edge", "tiny", "subnormal", "large", "zero",
                                  "one_tiny", "inf", "nan"])
def test_cells_outside_the_method_divide(sfg, kind, nx):
    """A uniform periodic field without forces: after a step every cell holds the
    collision of the one before, here computed with numpy's divisions."""
    import softflow_b200 as S
    rng = np.random.default_rng(8)
    f = W * (1 + 0.1 * rng.uniform(-1, 1, 9))
    scale = {"small": 1e-8, "edge": 2.0 ** -199, "tiny": 1e-70, "subnormal": 1e-310, "large": 1e100}
    f = f * scale.get(kind, 1.0)
    if kind == "zero":
        f[:] = [0.5, 0, 0, 0, 0, 0.25, 0, 0.25, 0]
    if kind in ("one_tiny", "inf", "nan"):
        f[3] = {"one_tiny": 1e-200, "inf": np.inf, "nan": np.nan}[kind]
    ens = S.Ensemble(precision="fp64")
    p = S.SimulationParams(nx=nx, ny=12, precision="fp64")
    p.fluid.boundary_type = S.BoundaryType.PERIODIC
    p.fluid.collision_model = S.CollisionModel.REGULARIZED
    p.fluid.tau = 0.8
    p.fluid.periodic_y = True
    i = ens.add_channel(p)
    ens.initialize()
    ens.field(i).set_distributions(np.broadcast_to(f[:, None, None], (9, 12, nx)))
    ens.run(1)
    got = ens.field(i).distributions()
    with np.errstate(all="ignore"):
        want = _regularized(f, 1.0 / 0.8)
    assert np.array_equal(got, np.broadcast_to(want[:, None, None], got.shape), equal_nan=True)


def _mrt(f, rates):
    """collide of the FP64 MRT cell without forces, numpy's divisions."""
    sn, s1, s2, s4 = rates
    r, vx, vy = _velocity(f)
    m = [f[0] + f[1] + f[2] + f[3] + f[4] + f[5] + f[6] + f[7] + f[8],
         -4 * f[0] - f[1] - f[2] - f[3] - f[4] + 2 * f[5] + 2 * f[6] + 2 * f[7] + 2 * f[8],
         4 * f[0] - 2 * f[1] - 2 * f[2] - 2 * f[3] - 2 * f[4] + f[5] + f[6] + f[7] + f[8],
         f[1] - f[3] + f[5] - f[6] - f[7] + f[8],
         -2 * f[1] + 2 * f[3] + f[5] - f[6] - f[7] + f[8],
         f[2] - f[4] + f[5] + f[6] - f[7] - f[8],
         -2 * f[2] + 2 * f[4] + f[5] + f[6] - f[7] - f[8],
         f[1] - f[2] + f[3] - f[4], f[5] - f[6] + f[7] - f[8]]
    uu = vx * vx + vy * vy
    eq = {1: -2 * r + 3 * r * uu, 2: r - 3 * r * uu, 4: -r * vx, 6: -r * vy,
          7: r * (vx * vx - vy * vy), 8: r * vx * vy}
    for k, s in ((1, s1), (2, s2), (4, s4), (6, s4), (7, sn), (8, sn)):
        m[k] = m[k] - s * (m[k] - eq[k]) + 0.0
    m0, m1, m2, m3, m4, m5, m6, m7, m8 = m
    return np.array([
        m0 / 9 - m1 / 9 + m2 / 9,
        m0 / 9 - m1 / 36 - m2 / 18 + m3 / 6 - m4 / 6 + m7 / 4,
        m0 / 9 - m1 / 36 - m2 / 18 + m5 / 6 - m6 / 6 - m7 / 4,
        m0 / 9 - m1 / 36 - m2 / 18 - m3 / 6 + m4 / 6 + m7 / 4,
        m0 / 9 - m1 / 36 - m2 / 18 - m5 / 6 + m6 / 6 - m7 / 4,
        m0 / 9 + m1 / 18 + m2 / 36 + m3 / 6 + m4 / 12 + m5 / 6 + m6 / 12 + m8 / 4,
        m0 / 9 + m1 / 18 + m2 / 36 - m3 / 6 - m4 / 12 + m5 / 6 + m6 / 12 - m8 / 4,
        m0 / 9 + m1 / 18 + m2 / 36 - m3 / 6 - m4 / 12 - m5 / 6 - m6 / 12 + m8 / 4,
        m0 / 9 + m1 / 18 + m2 / 36 + m3 / 6 + m4 / 12 - m5 / 6 - m6 / 12 - m8 / 4])


@pytest.mark.gpu
@pytest.mark.parametrize("nx", [64, 63])
@pytest.mark.parametrize("kind", ["plain", "edge", "tiny", "subnormal", "one_tiny", "inf", "rate"])
def test_mrt_cells_outside_the_method_divide(sfg, kind, nx):
    import softflow_b200 as S
    rng = np.random.default_rng(9)
    f = W * (1 + 0.1 * rng.uniform(-1, 1, 9))
    f = f * {"edge": 2.0 ** -199, "tiny": 1e-70, "subnormal": 1e-310}.get(kind, 1.0)
    if kind in ("one_tiny", "inf"):
        f[3] = {"one_tiny": 1e-200, "inf": np.inf}[kind]
    ens = S.Ensemble(precision="fp64")
    p = S.SimulationParams(nx=nx, ny=12, precision="fp64")
    p.fluid.boundary_type = S.BoundaryType.PERIODIC
    p.fluid.collision_model = S.CollisionModel.MRT
    p.fluid.tau = 0.8
    p.fluid.periodic_y = True
    if kind == "rate":
        p.fluid.mrt_se = 1e-290
        f = W.copy()   # moments that vanish, but for rounding
    i = ens.add_channel(p)
    ens.initialize()
    ens.field(i).set_distributions(np.broadcast_to(f[:, None, None], (9, 12, nx)))
    ens.run(1)
    got = ens.field(i).distributions()
    fl = p.fluid
    with np.errstate(all="ignore"):
        want = _mrt(f, (1.0 / 0.8, fl.mrt_se, fl.mrt_s_eps, fl.mrt_sq))
    assert np.array_equal(got, np.broadcast_to(want[:, None, None], got.shape), equal_nan=True)

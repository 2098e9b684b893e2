"""The per-marker kernels with four lanes a marker (contexts of at most 32,768
markers) and with one thread a marker (larger ones) compute the same sums in the
same order: a channel run alone, with few markers, equals the same channel inside
an ensemble on the other side of the line, bit for bit.  Marker counts end at
odd places of the warps and blocks on both sides."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _build(S, precision, n_copies, nodes):
    ens = S.Ensemble(precision=precision)
    for k in range(1 + n_copies):
        p = S.SimulationParams(nx=72 if k == 0 else 320, ny=44 if k == 0 else 200,
                               ibm_iterations=4, precision=precision)
        p.fluid.boundary_type = S.BoundaryType.PERIODIC
        p.fluid.collision_model = S.CollisionModel.BGK
        p.fluid.body_force_x = 2e-5
        i = ens.add_channel(p)
        mp = S.MembraneParams(model=S.MembraneModel.NEO_HOOKEAN, G_s=0.05)
        if k == 0:
            for c in ((1.2, 20.3), (30.4, 9.1), (52.8, 33.9)):     # seam, wall, interior
                ens.addCapsule(i, c, 4.0, nodes, mp)
        else:
            for cy in range(12, 190, 16):
                for cx in range(10, 316, 16):
                    ens.addCapsule(i, (cx, cy), 4.0, 32, mp)
    ens.initialize()
    return ens


@pytest.mark.parametrize("precision", ["fp64", "fp32", "fp16s"])
@pytest.mark.parametrize("nodes", [27, 33])
def test_few_and_many_markers_agree(sfg, precision, nodes):
    import softflow_b200 as S
    few, many = _build(S, precision, 0, nodes), _build(S, precision, 5, nodes)
    assert few.num_markers() <= 32768 < many.num_markers()
    few.run(6)
    many.run(6)
    for a, b in zip(few.field(0).macroscopic(), many.field(0).macroscopic()):
        assert np.array_equal(a, b)
    assert np.array_equal(few.capsules(0).positions(), many.capsules(0).positions())
    assert np.array_equal(few.capsules(0).velocities(), many.capsules(0).velocities())


@pytest.mark.parametrize("precision", ["fp32", "fp16s"])
@pytest.mark.parametrize("sweeps", [1, 4])
@pytest.mark.parametrize("nodes", [9, 33, 200])
def test_few_and_many_tiles_agree(sfg, precision, sweeps, nodes):
    """The FP32 spread gives a tile one warp, or four in contexts of at most 8,192
    tiles: again the same channel on both sides of that line, bit for bit.  The
    tiles' lists hold from a few markers to far more than one pass of four warps
    (32), and the tiles at the right and upper edge are partly outside."""
    import softflow_b200 as S
    ctx = []
    for many in (False, True):
        ens = S.Ensemble(precision=precision)
        for nx, ny in ((77, 43),) + (((1056, 2048),) if many else ()):
            p = S.SimulationParams(nx=nx, ny=ny, ibm_iterations=sweeps, precision=precision)
            p.fluid.boundary_type = S.BoundaryType.PERIODIC
            p.fluid.collision_model = S.CollisionModel.BGK
            p.fluid.body_force_x = 2e-5
            i = ens.add_channel(p)
            mp = S.MembraneParams(model=S.MembraneModel.NEO_HOOKEAN, G_s=0.05)
            if i == 0:
                for c in ((1.2, 20.3), (30.4, 9.1), (70.8, 33.9)):
                    ens.addCapsule(i, c, 4.0, nodes, mp)
            else:
                for k in range(40):
                    ens.addCapsule(i, (20 + 25 * k, 40 + 45 * k), 4.0, 32, mp)
        ens.initialize()
        ens.run(5)
        ctx.append(ens)
    few, many = ctx
    for a, b in zip(few.field(0).macroscopic(), many.field(0).macroscopic()):
        assert np.isfinite(a).all() and np.array_equal(a, b)
    assert np.array_equal(few.capsules(0).positions(), many.capsules(0).positions())
    assert np.array_equal(few.capsules(0).velocities(), many.capsules(0).velocities())


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("nodes", [12, 80])
def test_crowded_contact_agrees(sfg, precision, nodes):
    """Capsules whose membranes touch: a lane of a marker's four keeps up to four
    forces that are not zero, and with 80 nodes a capsule far more lie within the
    cut-off, so that one thread adds them; alone and among many markers alike."""
    import softflow_b200 as S
    out = []
    for n_many in (0, 5):
        ens = S.Ensemble(precision=precision)
        for k in range(1 + n_many):
            p = S.SimulationParams(nx=72 if k == 0 else 320, ny=44 if k == 0 else 200,
                                   ibm_iterations=1, precision=precision)
            p.fluid.boundary_type = S.BoundaryType.PERIODIC
            p.fluid.collision_model = S.CollisionModel.BGK
            i = ens.add_channel(p)
            mp = S.MembraneParams(model=S.MembraneModel.NEO_HOOKEAN, G_s=0.05)
            if k == 0:
                # a touching pair across the seam, one capsule at the wall
                for c in ((2.0, 20.3), (68.0, 21.1), (30.4, 6.2)):
                    ens.addCapsule(i, c, 4.0, nodes, mp)
            else:
                for cy in range(12, 190, 16):
                    for cx in range(10, 316, 16):
                        ens.addCapsule(i, (cx, cy), 4.0, 32, mp)
        ens.initialize()
        a, b = (ens.capsules(0).positions().reshape(-1, 2)[k * nodes:(k + 1) * nodes]
                for k in (0, 1))
        d = a[:, None] - b[None]
        d[..., 0] -= 72 * np.round(d[..., 0] / 72)
        near = (np.hypot(d[..., 0], d[..., 1]) < p.repulsion.r_cut).sum(1).max()
        assert 0 < near if nodes == 12 else near > 16   # more than four lanes keep
        ens.run(2)
        out.append((ens.num_markers(), ens.capsules(0).positions().copy(),
                    ens.capsules(0).velocities().copy()))
    assert out[0][0] <= 32768 < out[1][0]
    for x, y in zip(out[0][1:], out[1][1:]):
        assert np.isfinite(x).all() and np.array_equal(x, y)


@pytest.mark.parametrize("nx,ny,r,nodes,sweeps", [
    (9, 24, 2.0, 12, 3),        # narrower than a stencil's residues, over the seam
    (32, 24, 4.0, 24, 2),       # one tile wide
    (33, 24, 4.0, 24, 2),       # a second tile of one column
    (77, 43, 4.0, 9, 4), (77, 43, 4.0, 150, 1), (77, 43, 4.0, 150, 4),
    (77, 43, 3.0, 600, 3),      # lists beyond 256 entries
])
def test_fp64_few_and_many_touched_tiles_agree(sfg, nx, ny, r, nodes, sweeps):
    """The FP64 spread gives a tile four warps, or one in contexts whose markers touch
    more than 2,800 tiles: the same channel on both sides of that line, bit for bit."""
    import softflow_b200 as S
    ctx = []
    for many in (False, True):
        ens = S.Ensemble(precision="fp64")
        for w, h in ((nx, ny),) + (((2048, 512),) if many else ()):
            p = S.SimulationParams(nx=w, ny=h, ibm_iterations=sweeps, precision="fp64")
            p.fluid.boundary_type = S.BoundaryType.PERIODIC
            p.fluid.collision_model = S.CollisionModel.BGK
            p.fluid.body_force_x = 2e-5
            i = ens.add_channel(p)
            mp = S.MembraneParams(model=S.MembraneModel.NEO_HOOKEAN, G_s=0.05)
            if i == 0:
                for c in ((1.2, 11.3),) + (((30.4, 12.1), (70.8, 30.9)) if nx > 40 else ()):
                    ens.addCapsule(i, c, r, nodes, mp)
            else:
                for cy in range(10, 505, 16):
                    for cx in range(10, 2040, 16):
                        ens.addCapsule(i, (cx, cy), 4.0, 12, mp)
        ens.initialize()
        ens.run(3)
        ctx.append(ens)
    few, many = ctx
    for a, b in zip(few.field(0).macroscopic(), many.field(0).macroscopic()):
        assert np.isfinite(a).all() and np.array_equal(a, b)
    assert np.array_equal(few.capsules(0).positions(), many.capsules(0).positions())
    assert np.array_equal(few.capsules(0).velocities(), many.capsules(0).velocities())

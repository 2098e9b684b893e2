"""The marker move of the FP32-arithmetic modes, whose velocity comes from the
capsule's box of cells in shared memory, or cell by cell where the box is larger:
after a step, each marker's velocity is the field's, interpolated in double at the
position it had.

Tolerance: the moments of a cell are sums of nine FP32 populations of at most 1
(9 x 6e-8 at most, some 5e-7), the weights and the 16-term sum add a relative
20 x 6e-8 of a velocity below 0.1; 2e-6 in all.  One cell beside the right one is
1e-3 off (the velocity's slope near the walls), as is a lost force or weight."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp16s"])
@pytest.mark.parametrize("r,nodes", [(3.0, 24), (9.0, 30), (9.5, 130), (14.0, 90)])
def test_velocity_is_the_interpolated_field(sfg, oracle_mod, precision, r, nodes):
    import oracle as O
    import softflow_b200 as S
    nx, ny = 131, 67
    sim = S.Ensemble(precision=precision)
    p = S.SimulationParams(nx=nx, ny=ny, ibm_iterations=1, precision=precision)
    p.fluid.boundary_type = S.BoundaryType.PERIODIC
    p.fluid.collision_model = S.CollisionModel.BGK
    p.fluid.body_force_x = 5e-4
    i = sim.add_channel(p)
    mp = S.MembraneParams(model=S.MembraneModel.NEO_HOOKEAN, G_s=0.001)
    for c in ((1.3, 18.2), (64.9, 46.7)):          # over the seam, inside
        sim.addCapsule(i, c, r, nodes, mp)
    sim.initialize()
    sim.run(40)
    pos = sim.capsules(i).positions().reshape(-1, 2).copy()
    sim.run(1)
    _, ux, uy, _, _ = (np.asarray(a) for a in sim.field(i).macroscopic())
    vel = sim.capsules(i).velocities().reshape(-1, 2)
    want = np.zeros_like(vel)
    for m, (x, y) in enumerate(pos):
        ix, iy = int(np.floor(x)), int(np.floor(y))
        for jy in range(iy - 1, iy + 3):
            for jx in range(ix - 1, ix + 3):
                w = O.phi(x - jx, "sfo") * O.phi(y - jy, "sfo")
                want[m] += w * np.array([ux[jy, jx % nx], uy[jy, jx % nx]])
    assert np.abs(want[:, 0]).max() > 1e-2
    assert np.abs(vel - want).max() < 2e-6

"""The step's marker lists (contact cells, force-tile slots and lists) at the
sizes where their construction changes: just above the all-pairs limit of 100
markers, cells of more than 32 markers (sorted in place instead of in
thread-local memory), marker counts around a block of 256, and tile counts that
are no multiple of a warp.  FP64 against the oracle: the pair counts are
integers, forces differ only by the device pow of the contact law (1e-8
relative, as the coupled parity tests)."""
import numpy as np
import pytest

import oracle as O
from cases import build_gpu, build_oracle, rel_l2

pytestmark = pytest.mark.gpu


def _case(nx, ny, rings, sweeps=2):
    return dict(spec=dict(nx=nx, ny=ny, collision=O.BGK, tau=0.8, body_fx=2e-5,
                          ibm_iterations=sweeps),
                capsules=[("add", cx, cy, r, n, dict(model=O.NEO_HOOKEAN, G_s=0.05))
                          for cx, cy, r, n in rings], conc=None)


@pytest.mark.parametrize("nx,ny,rings", [
    (64, 40, [(20.3, 19.7, 3.0, 50), (27.9, 20.4, 3.0, 51)]),       # 101 markers: cell list
    (64, 40, [(20.3, 19.7, 2.0, 64), (23.1, 20.4, 2.0, 64), (21.7, 23.0, 2.0, 64)]),
    (64, 40, [(20.3, 19.7, 1.5, 160), (23.6, 20.4, 1.5, 160)]),     # crowded cells
    (200, 33, [(8.0 + 16 * k, 16.2, 3.0, 32) for k in range(8)]),   # 256 markers, 35 tiles
    (201, 41, [(8.0 + 16 * k, 16.2 + (k % 3), 3.0, 33) for k in range(8)]),
    (37, 26, [(36.5, 12.0, 3.0, 60), (8.0, 13.0, 3.0, 60)]),        # across the seam
])
def test_lists_against_oracle(sfg, oracle_mod, nx, ny, rings):
    case = _case(nx, ny, rings)
    o = build_oracle(case)
    sim = build_gpu(case, "fp64")
    for _ in range(3):          # the records must be empty again for the next step
        o.step(1)
        sim.run(1)
        assert np.array_equal(sim.capsules().contact_counts(), o.contact_pairs()[0])
        assert rel_l2(sim.capsules().forces(), o.forces()) < 1e-8
        assert np.max(np.abs(sim.capsules().positions() - o.positions())) < 1e-9
        assert rel_l2(sim.field().force_x(), o.Fx()) < 1e-8


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("r_cut,n", [(3.5, 160), (9.0, 64), (25.0, 64)])
def test_cells_of_many_markers_against_oracle(sfg, oracle_mod, precision, r_cut, n):
    """Cells of more than 12 markers, ranked by a warp, and of several capsules each,
    where a marker's lane finds far more than four forces; few markers (four lanes each)
    and, with a second channel, many (one thread).  Pair counts are integers; forces
    in the tolerances of the other cases (FP32 keeps positions and contact in double)."""
    import softflow_b200 as S
    from cases import add_case_capsules, gpu_params
    case = _case(96, 60, [(14.0 + 17 * k, 20.3 + 16 * j, 6.0, n)
                          for k in range(5) for j in range(2)], 1)
    case["spec"].update(rep_r_cut=r_cut, rep_epsilon=1e-4)
    o = build_oracle(case)
    o.step(1)
    for copies in (0, 4):
        ens = S.Ensemble(precision=precision)
        ens.add_channel(gpu_params(case, precision))
        add_case_capsules(ens, 0, case)
        for _ in range(copies):
            p = S.SimulationParams(nx=1024, ny=128, precision=precision)
            p.fluid.boundary_type = S.BoundaryType.PERIODIC
            j = ens.add_channel(p)
            mp = S.MembraneParams(model=S.MembraneModel.NEO_HOOKEAN, G_s=0.05)
            for cy in range(16, 120, 20):
                for cx in range(16, 1010, 20):
                    ens.addCapsule(j, (cx, cy), 4.0, 34, mp)
        ens.initialize()
        ens.run(1)
        assert np.array_equal(ens.capsules(0).contact_counts(), o.contact_pairs()[0])
        assert rel_l2(ens.capsules(0).forces(), o.forces()) < 1e-8

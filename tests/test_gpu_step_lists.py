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

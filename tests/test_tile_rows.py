"""Tile rows of a marker's stencil: inside the channel's tiles for every stencil
that a step accepts, also where its rows lie beyond the lattice (a channel periodic
in y does not hold markers back there), and those of the rows inside.  On the
CPU the header the kernels use, compiled and run over every case; on the GPU a
capsule over the upper edge of a 16-row channel, whose markers reach the last
accepted position, against the oracle."""
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "softflow_b200", "csrc")

PROGRAM = r"""
#include "tile_rows.h"
#include <cstdio>
using namespace sfg;
int main() {
    for (int ny = 3; ny <= 200; ++ny) {
        const int tiles = (ny + TILE_H - 1) / TILE_H;
        for (int iy0 = -2; iy0 <= ny + 1; ++iy0) {      // the stencils a step accepts
            const int a = first_tile_row(iy0, ny), b = last_tile_row(iy0, ny);
            int lo = -1, hi = -1;
            for (int iy = iy0 - 1; iy <= iy0 + 2; ++iy)
                if (iy >= 0 && iy < ny) {
                    if (lo < 0) lo = iy / TILE_H;
                    hi = iy / TILE_H;
                }
            const bool in = a >= 0 && a < tiles && b >= 0 && b < tiles;
            if (!in || (lo >= 0 && (a != lo || b != hi))) {
                std::printf("ny %d iy0 %d: %d %d of %d tiles, rows inside in %d %d\n", ny, iy0,
                            a, b, tiles, lo, hi);
                return 1;
            }
        }
    }
    return 0;
}
"""


def test_rows_lie_inside_the_channel(tmp_path):
    src, exe = tmp_path / "rows.cpp", tmp_path / "rows"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 1e-5)])
@pytest.mark.parametrize("ny", [16, 19])
def test_markers_beyond_the_upper_edge(sfg, oracle_mod, ny, precision, tol):
    """Few markers and, with a second channel, many (four lanes a marker, one thread).
    Tolerances: FP64 follows the oracle's order; FP32 moves a marker by velocities below
    1e-2 with a relative error below 1e-4 over three steps of coordinates near ny."""
    import oracle as O
    from cases import add_case_capsules, build_oracle, gpu_params
    import softflow_b200 as S
    case = dict(spec=dict(nx=48, ny=ny, collision=O.BGK, tau=0.8, body_fx=2e-5, periodic_y=1,
                          ibm_iterations=2),
                capsules=[("add", 20.3, ny - 1.1, 2.9, 24, dict(model=O.NEO_HOOKEAN, G_s=0.05))],
                conc=None)
    o = build_oracle(case)
    assert o.positions().reshape(-1, 2)[:, 1].max() >= ny + 1.0
    o.step(3)
    for copies in (0, 4):
        ens = S.Ensemble(precision=precision)
        ens.add_channel(gpu_params(case, precision))
        add_case_capsules(ens, 0, case)
        for k in range(copies):
            p = S.SimulationParams(nx=1024, ny=128, ibm_iterations=2, precision=precision)
            p.fluid.boundary_type = S.BoundaryType.PERIODIC
            j = ens.add_channel(p)
            mp = S.MembraneParams(model=S.MembraneModel.NEO_HOOKEAN, G_s=0.05)
            for cy in range(16, 120, 20):
                for cx in range(16, 1010, 20):
                    ens.addCapsule(j, (cx, cy), 4.0, 34, mp)
        ens.initialize()
        ens.run(3)
        assert np.abs(ens.capsules(0).positions() - o.positions()).max() < tol

"""The tiled finite-difference steps at the edges of tiles, launches and speed
checks, against the CPU restatement: the tolerance of test_gpu_fdtd, 1e-9 of
the largest sample."""
import pathlib
import sys

import numpy as np
import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT / "oracle"))
import fdtd_oracle as FO  # noqa: E402

pytestmark = pytest.mark.gpu

LAYERED = [(2.0, 350.0, 140.0, 1600.0), (0.0, 800.0, 320.0, 2000.0)]


@pytest.mark.parametrize("lossy", [False, True])
@pytest.mark.parametrize("max_range,depth,pml,steps", [
    (0.9, 0.6, 2, 1),      # a few cells, one step
    (2.0, 1.4, 3, 37),     # smaller than a window
    (6.2, 2.6, 4, 258),    # one step past the second speed check
    (12.6, 6.4, 20, 120),  # several tiles each way, damped columns across a tile edge
    (5.0, 17.0, 5, 60),    # narrow and deep
])
def test_tiles_against_oracle(gfk, engine, lossy, max_range, depth, pml, steps):
    sls = gfk.SLS.fit(25, 30) if lossy else None
    stack = gfk.Stack([gfk.Layer(h, vp, vs, rho, 0, 0) for h, vp, vs, rho in LAYERED])
    md = gfk.fdtd.Model(stack, relax=sls, ref_freq=30, max_range=max_range, depth=depth, spacing=0.2, pml_cells=pml,
                        dominant_freq=25)
    dt = md.grid()[0]
    force = gfk.fdtd.ricker(1000, 25, dt, steps)
    ranges = np.arange(0.0, max_range - 0.2, 0.2).tolist()  # every interior column: each tile's first and last
    res = gfk.fdtd.run(gfk.fdtd.Shot(md, force, ranges, steps), engine=engine)
    sim = FO.Sim(LAYERED, FO.SLS.fit(25, 30) if lossy else None, 30, max_range, depth, 0.2, pml_cells=pml,
                 dominant_freq=25)
    assert (sim.nr, sim.nz) == res.cells
    want = FO.run(sim, FO.ricker(1000, 25, dt, steps), ranges, steps)
    got = np.array([t.vertical for t in res.traces])
    assert np.abs(got - want).max() <= 1e-9 * np.abs(want).max()

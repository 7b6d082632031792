"""The closed-form layer step of the secular function in each of its regimes,
against the CPU restatement (scipy expm): the tolerance of test_gpu_disp,
1e-9 max(1, |F|); and the scan in chunks of frequencies."""
import pathlib
import sys

import numpy as np
import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT / "oracle"))
import disp_oracle as D  # noqa: E402

pytestmark = pytest.mark.gpu


def stack(gfk, layers):
    return gfk.Stack([gfk.Layer(h, vp, vs, rho, 20, 40) for h, vp, vs, rho in layers])


@pytest.mark.parametrize("h", [1e-3, 0.05, 0.4, 2.0])
def test_secular_in_every_regime(gfk, engine, h):
    """k h from 1e-4 to 40: power series; a stiff layer (c far below its
    velocities: eigenvalues a quarter apart or less); propagating and decaying
    P and S waves, and the velocities where one turns into the other."""
    layers = [(h, 300.0, 150.0, 1500.0), (0.7 * h, 2800.0, 1500.0, 2300.0), (1.9 * h, 500.0, 260.0, 1900.0),
              (0.0, 2000.0, 1000.0, 2200.0)]
    rng = np.random.default_rng(int(h * 1000))
    f = np.concatenate([rng.uniform(0.5, 300.0, 36), [20.0] * 5])
    c = np.concatenate([rng.uniform(128.0, 999.0, 36), [150.0, 260.0, 300.0, 500.0, 999.9]])
    v, ok = gfk.disp.secular_at_velocity(stack(gfk, layers), f, c, engine=engine)
    for i in range(len(f)):
        w = D.secular_at_velocity(layers, f[i], c[i])
        assert ok[i] == (w is not None)
        if w is not None:
            assert abs(v[i] - w) <= 1e-9 * max(1.0, abs(w)), (f[i], c[i], v[i], w)


def test_scan_in_chunks_gives_the_same_modes(gfk, engine):
    """5000 frequencies need two chunks of scan values; 16384 samples make a
    chunk of a few hundred; one frequency at a time has the same roots."""
    st = stack(gfk, [(3.0, 400.0, 160.0, 1600.0), (0.0, 900.0, 400.0, 2000.0)])
    f = np.linspace(1.0, 140.0, 5000)
    many = gfk.disp.modes_many(st, f, engine=engine)
    for i in (0, 1, 4090, 4095, 4096, 4999):
        assert gfk.disp.modes(st, f[i], engine=engine) == many[i]
    fine = gfk.disp.Search(16384)
    few = gfk.disp.modes_many(st, f[::7], fine, engine=engine)
    for i in (0, 500, 520, 714):
        assert gfk.disp.modes(st, f[::7][i], fine, engine=engine) == few[i]

"""Banks of 1 to 8 ranges on a shared grid: short rows and small plans solve every
wavenumber inside the fused sum, others (and a forced launch shape) panels' nodes. Both
against the CPU oracle, rel-L2 <= 1e-9 per frequency as in test_gpu_panels, at the
lines between the launches; what the plan says of its launch; and weights that plans of
both kinds share."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu
SOIL = [(0.8, 240.0, 120.0, 1600.0, 10.0, 20.0), (0.8, 480.0, 240.0, 1750.0, 30.0, 60.0),
        (0.8, 800.0, 400.0, 1900.0, 45.0, 90.0), (0.0, 1200.0, 600.0, 2100.0, 60.0, 120.0)]
RUNS = {68: 1, 69: 2, 70: 9, 71: 8, 72: 8}


def medium(gfk, engine, layers):
    return gfk.Medium(gfk.Stack(gfk.Layer(*t) for t in SOIL[-layers:]), formulation=gfk.DUNKIN, omega_imag=0.8,
                      engine=engine)


def execute(gfk, engine, m, ranges, freqs, nk, kmax=40.0):
    p = gfk.Plan(m, ranges, freqs, gfk.Integration(nk, 0.0, kmax), engine=engine)
    p.execute()
    got, status = p.download()
    assert (status == 0).all()
    shape = p.prop_shape()
    p.close()
    assert shape["runs_per_item"] == RUNS[shape["index"]] and shape["blocks_per_sm"] == (6 if shape["index"] == 71 else 4)
    return got, shape["index"]


@pytest.mark.parametrize("nr", [1, 2, 3, 8])
@pytest.mark.parametrize("layers,nf,nk,want", [
    (4, 1, 1, 68), (4, 5, 127, 68), (4, 5, 129, 68), (4, 147, 70, 68), (4, 148, 256, 70), (4, 399, 257, 68), (4, 400, 257, 70),
    (3, 4, 1152, 68), (3, 4, 1153, 69), (3, 4, 1281, 69), (4, 4, 1153, 68), (1, 3, 2500, 69), (1, 40, 3750, 69),
    (1, 40, 3751, None), (1, 2, 4096, 69), (1, 2, 4097, None), (4, 2, 10240, 68), (4, 2, 10241, None),
])
def test_direct_sums_against_oracle(gfk, engine, oracle, nr, layers, nf, nk, want):
    freqs, ranges = np.linspace(7.0, 260.0, nf), np.linspace(1.0, 21.0, nr)
    got, index = execute(gfk, engine, medium(gfk, engine, layers), ranges, freqs, nk)
    assert index == (want or (71 if nr <= 2 else 72))
    ref, ost = oracle.bank_spectra(SOIL[-layers:], ranges, freqs, samples=nk, kmax=40.0, formulation=oracle.DUNKIN,
                                   omega_imag=0.8)
    assert (ost == 0).all()
    assert max(rel_l2(g, w) for g, w in zip(got, ref)) < 1e-9


@pytest.mark.parametrize("nf,nk,want", [(390, 1153, 69), (391, 1153, None), (2000, 1000, 70)])
def test_direct_and_panels_agree(gfk, engine, monkeypatch, nf, nk, want):
    m, freqs, ranges = medium(gfk, engine, 3), np.linspace(5.0, 240.0, nf), np.array([2.0, 5.0, 11.0])
    got, index = execute(gfk, engine, m, ranges, freqs, nk)
    assert index == (want or 72)
    monkeypatch.setenv("GFK_PROP_VARIANT", "0")
    forced, index = execute(gfk, engine, m, ranges, freqs, nk)
    assert index == 72
    if want is None:
        assert np.array_equal(got, forced)
    assert max(rel_l2(g, w) for g, w in zip(got, forced)) <= 1e-9


def test_shared_weights(gfk, engine, monkeypatch):
    """A direct plan builds the Hankel weights alone; a plan of panels on the same
    grid then adds its node weights, and either kind still has its own."""
    m, ranges = medium(gfk, engine, 4), np.array([1.5, 6.0])
    few, many = np.array([30.0]), np.linspace(5.0, 240.0, 300)
    before = engine.kernel_launches()
    a, index = execute(gfk, engine, m, ranges, few, 2100, 40.125)
    assert index == 68 and engine.kernel_launches() - before == 5  # layers, statics, weights, sum, finish
    b, index = execute(gfk, engine, m, ranges, many, 2100, 40.125)
    assert index == 71
    assert np.array_equal(execute(gfk, engine, m, ranges, few, 2100, 40.125)[0], a)
    assert np.array_equal(execute(gfk, engine, m, ranges, many, 2100, 40.125)[0], b)
    at = execute(gfk, engine, m, ranges, np.append(few, many), 2100, 40.125)[0]
    assert rel_l2(at[0], a[0]) <= 1e-9 and max(rel_l2(g, w) for g, w in zip(at[1:], b)) <= 1e-9

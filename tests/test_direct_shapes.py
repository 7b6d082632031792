"""The propagator launches that solve every wavenumber: which plans take them, what
the plan says of its launch, and their banks against the panels that a forced launch
shape takes (rel-L2 per frequency as in test_gpu_direct_points)."""
import numpy as np
import pytest

from conftest import rel_l2

SOIL = [(0.8, 240.0, 120.0, 1600.0, 10.0, 20.0), (0.8, 480.0, 240.0, 1750.0, 30.0, 60.0),
        (0.0, 1200.0, 600.0, 2100.0, 60.0, 120.0)]
FEW, MANY, ROW = ({"threads": 128, "blocks_per_sm": b, "wavenumbers_per_thread": 1, "runs_per_item": r,
                   "persistent": False} for b, r in ((4, 1), (5, 1), (5, 9)))


def test_described_without_a_gpu(gfk):
    assert [gfk.prop_shape(64 + i) for i in range(3)] == [dict(d, index=64 + i) for i, d in enumerate((FEW, MANY, ROW))]
    for v in (63, 1000):
        with pytest.raises(gfk.FkError):
            gfk.prop_shape(v)


# rows x wavenumbers on both sides of: a short row (1152), many of them (444), 15 runs of 128
# an SM (2220), one long item for 240 half-space rows, 950000 points; beyond the smallest
@pytest.mark.gpu
@pytest.mark.parametrize("layers,nf,nk,want", [
    (3, 1, 1, FEW), (3, 443, 129, FEW), (3, 444, 128, FEW), (3, 444, 129, ROW), (3, 444, 1152, ROW), (3, 222, 1280, FEW), (3, 223, 1153, MANY),
    (3, 443, 1152, MANY), (1, 119, 2304, FEW), (1, 120, 2304, ROW), (3, 900, 1152, ROW), (3, 2100, 1000, ROW),
    (3, 823, 1154, MANY), (3, 824, 1153, None), (1, 824, 1153, None),
])
@pytest.mark.parametrize("split", [False, True])
def test_plans_say_what_ran(gfk, engine, monkeypatch, layers, nf, nk, want, split):
    m = gfk.Medium(gfk.Stack(gfk.Layer(*t) for t in SOIL[-layers:]), formulation=gfk.DUNKIN, omega_imag=0.8,
                   engine=engine, quadrature=gfk.SPLIT_INT8 if split else gfk.PLAIN_FP64)
    freqs, ranges, opt = np.linspace(5.0, 240.0, nf), np.linspace(1.0, 21.0, 9), gfk.Integration(nk, 0.0, 40.0)
    banks = []
    for force in (False, True):
        if force:
            monkeypatch.setenv("GFK_PROP_VARIANT", "2")
        p = gfk.Plan(m, ranges, freqs, opt, engine=engine)
        p.execute()
        shape = p.prop_shape()
        if nf == 1 and not split:  # one row is a per-frequency grid: 8 panels a block, whatever is forced
            assert shape == gfk.prop_shape(1) and shape["runs_per_item"] == 8
        elif force or want is None:
            assert shape["index"] < 64
        else:
            assert {k: v for k, v in shape.items() if k != "index"} == want
        got, status = p.download()
        assert (status == 0).all()
        banks.append(got)
        p.close()
    tol = 1e-6 if split else 1e-9
    assert max(rel_l2(g, w) for g, w in zip(*banks)) <= tol

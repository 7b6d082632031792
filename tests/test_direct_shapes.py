"""The propagator launches that solve every wavenumber: which plans take them, what
the plan says of its launch, and their banks against the panels that a forced launch
shape takes (rel-L2 per frequency as in test_gpu_direct_points)."""
import numpy as np
import pytest

from conftest import rel_l2

SOIL = [(0.8, 240.0, 120.0, 1600.0, 10.0, 20.0), (0.8, 480.0, 240.0, 1750.0, 30.0, 60.0),
        (0.0, 1200.0, 600.0, 2100.0, 60.0, 120.0)]
FEW, MANY, ROW, PAIR = ({"threads": t, "blocks_per_sm": b, "wavenumbers_per_thread": 1, "runs_per_item": r,
                         "persistent": False} for t, b, r in ((128, 4, 1), (128, 5, 1), (128, 5, 9), (256, 2, 1)))


def test_described_without_a_gpu(gfk):
    assert [gfk.prop_shape(64 + i) for i in range(4)] == [dict(d, index=64 + i)
                                                        for i, d in enumerate((FEW, MANY, ROW, PAIR))]
    for v in (63, 1000):
        with pytest.raises(gfk.FkError):
            gfk.prop_shape(v)


# rows x wavenumbers on both sides of: rows of one run of 128 (592, 740, 1184 of them), of two (296
# rows), short rows (400 up to 512, then 1000 plain or 540 split, up to 1152), four runs plain (592,
# 1184), one long item for 240 half-space rows, 444 and 1924 runs of long rows split, 1184 runs,
# 950000 points; a pair (plain, split) where the sum matters; beyond the smallest
@pytest.mark.gpu
@pytest.mark.parametrize("layers,nf,nk,want", [
    (3, 1, 1, FEW), (3, 592, 128, FEW), (3, 593, 128, MANY), (3, 740, 70, MANY), (3, 741, 128, FEW), (3, 1184, 99, FEW),
    (3, 1185, 128, MANY), (3, 296, 129, PAIR), (3, 297, 129, ROW), (3, 296, 256, PAIR), (3, 297, 255, ROW),
    (3, 394, 257, FEW), (3, 399, 257, MANY), (3, 400, 257, ROW), (3, 148, 512, FEW), (3, 149, 512, (PAIR, FEW)),
    (3, 296, 385, (PAIR, FEW)), (3, 297, 512, MANY), (3, 539, 513, MANY), (3, 540, 1152, (MANY, ROW)), (3, 540, 513, (MANY, ROW)),
    (3, 999, 1000, (MANY, ROW)), (3, 1000, 1152, ROW), (1, 119, 2304, MANY), (1, 120, 2304, ROW), (3, 26, 2049, FEW),
    (3, 27, 2049, (FEW, PAIR)), (3, 60, 2048, FEW), (3, 113, 2049, (MANY, PAIR)), (3, 114, 2049, MANY), (3, 74, 2048, FEW),
    (3, 75, 2048, MANY), (3, 2100, 1000, ROW), (3, 823, 1154, MANY), (3, 824, 1153, None), (1, 824, 1153, None),
])
@pytest.mark.parametrize("split", [False, True])
def test_plans_say_what_ran(gfk, engine, monkeypatch, layers, nf, nk, want, split):
    m = gfk.Medium(gfk.Stack(gfk.Layer(*t) for t in SOIL[-layers:]), formulation=gfk.DUNKIN, omega_imag=0.8,
                   engine=engine, quadrature=gfk.SPLIT_INT8 if split else gfk.PLAIN_FP64)
    freqs, ranges, opt = np.linspace(5.0, 240.0, nf), np.linspace(1.0, 21.0, 9), gfk.Integration(nk, 0.0, 40.0)
    want = want[split] if isinstance(want, tuple) else want
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

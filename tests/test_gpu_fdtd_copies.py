"""Finite-difference steps with one copy of the fields (one launch per phase, in place)
beside those with two (tiles): each against the CPU restatement, 1e-9 of the largest
sample as in test_gpu_fdtd, and which of the two a shot takes."""
import pathlib
import sys

import numpy as np
import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT / "oracle"))
import fdtd_oracle as FO  # noqa: E402

pytestmark = pytest.mark.gpu

LAYERED = [(2.0, 350.0, 140.0, 1600.0), (0.0, 800.0, 320.0, 2000.0)]


def shot(gfk, max_range, depth, pml, steps, ranges, lossy=True):
    stack = gfk.Stack([gfk.Layer(h, vp, vs, rho, 0, 0) for h, vp, vs, rho in LAYERED])
    md = gfk.fdtd.Model(stack, relax=gfk.SLS.fit(25, 30) if lossy else None, ref_freq=30, max_range=max_range, depth=depth,
                        spacing=0.2, pml_cells=pml, dominant_freq=25)
    return gfk.fdtd.Shot(md, gfk.fdtd.ricker(1000, 25, md.grid()[0], steps), ranges, steps)


def traces(gfk, engine, s):
    """The traces, the largest speed and the launches of one run."""
    before = engine.kernel_launches()
    res = gfk.fdtd.run(s, engine=engine)
    return np.array([t.vertical for t in res.traces]), res.peak, engine.kernel_launches() - before


def per_phase(steps):
    return 2 * steps + (steps + 255) // 256  # two phases a step, a speed check at 0, 256, ...


@pytest.mark.parametrize("lossy", [False, True])
@pytest.mark.parametrize("max_range,depth,pml,steps", [
    (0.9, 0.6, 2, 1), (2.0, 1.4, 3, 37), (6.2, 2.6, 4, 258), (12.6, 6.4, 20, 120),
])
def test_one_copy_and_two(gfk, engine, monkeypatch, lossy, max_range, depth, pml, steps):
    ranges = np.arange(0.0, max_range - 0.2, 0.2).tolist()
    s = shot(gfk, max_range, depth, pml, steps, ranges, lossy)
    sim = FO.Sim(LAYERED, FO.SLS.fit(25, 30) if lossy else None, 30, max_range, depth, 0.2, pml_cells=pml, dominant_freq=25)
    want = FO.run(sim, s.force, ranges, steps)
    got = {}
    for copies in ("1", "2"):
        monkeypatch.setenv("GFK_FDTD_COPIES", copies)
        v, got[copies], launches = traces(gfk, engine, s)
        assert np.abs(v - want).max() <= 1e-9 * np.abs(want).max()
        assert (launches == per_phase(steps)) == (copies == "1")
    assert abs(got["1"] - got["2"]) <= 1e-9 * got["1"]


def test_one_copy_where_two_cannot_be_had(gfk, engine, monkeypatch):
    """A memory pool that holds one copy of the fields (115 MB) and not two."""
    drv = pytest.importorskip("cuda.bindings.driver")

    def ok(r):
        assert r[0] == drv.CUresult.CUDA_SUCCESS, r[0]
        return r[1] if len(r) > 1 else None

    s = shot(gfk, 196.0, 156.0, 20, 12, [0.0, 5.0, 40.0])
    monkeypatch.setenv("GFK_FDTD_COPIES", "1")
    want, peak, launches = traces(gfk, engine, s)
    assert launches == per_phase(12)
    monkeypatch.delenv("GFK_FDTD_COPIES")
    assert traces(gfk, engine, s)[2] < launches
    dev = ok(drv.cuCtxGetDevice())
    props = drv.CUmemPoolProps()
    props.allocType = drv.CUmemAllocationType.CU_MEM_ALLOCATION_TYPE_PINNED
    props.location.type = drv.CUmemLocationType.CU_MEM_LOCATION_TYPE_DEVICE
    props.location.id = int(dev)
    props.maxSize = 192 << 20
    pool, old = ok(drv.cuMemPoolCreate(props)), ok(drv.cuDeviceGetMemPool(dev))
    ok(drv.cuDeviceSetMemPool(dev, pool))
    try:
        got, peak1, launches1 = traces(gfk, engine, s)
    finally:
        ok(drv.cuDeviceSetMemPool(dev, old))
        ok(drv.cuMemPoolDestroy(pool))
    assert launches1 == launches and peak1 == peak and np.array_equal(got, want)

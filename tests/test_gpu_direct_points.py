"""Small banks solve every wavenumber, larger ones panels' nodes: both sides of the
line against each other (rel-L2 <= 1e-9 per frequency, as in test_gpu_parity),
and the panels of small banks, which a forced launch shape still takes, against
the CPU oracle at counts on both sides of the shortest panel and of an item."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu
SOIL = [(0.8, 240.0, 120.0, 1600.0, 10.0, 20.0), (0.8, 480.0, 240.0, 1750.0, 30.0, 60.0),
        (0.0, 1200.0, 600.0, 2100.0, 60.0, 120.0)]


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("nf,nk", [(1, 1), (3, 129), (95, 10000), (95, 10001)])  # 950000 is the last direct count
def test_direct_and_panels_agree(gfk, engine, monkeypatch, nf, nk, split):
    m = gfk.Medium(gfk.Stack(gfk.Layer(*t) for t in SOIL), formulation=gfk.DUNKIN, omega_imag=0.8, engine=engine,
                   quadrature=gfk.SPLIT_INT8 if split else gfk.PLAIN_FP64)
    freqs, ranges = np.linspace(5.0, 240.0, nf), np.linspace(1.0, 21.0, 9)
    opt = gfk.Integration(nk, 0.0, 40.0)
    got, status = m.bank_spectra(ranges, freqs, opt)
    assert (status == 0).all()
    monkeypatch.setenv("GFK_PROP_VARIANT", "2")
    forced, status = m.bank_spectra(ranges, freqs, opt)
    assert (status == 0).all()
    if nf * nk > 950000:
        assert np.array_equal(got, forced)
    tol = 1e-6 if split else 1e-9
    assert max(rel_l2(g, w) for g, w in zip(got, forced)) <= tol


@pytest.mark.parametrize("nk", [64, 97, 161, 1057])
def test_panels_of_a_small_bank_against_oracle(gfk, engine, oracle, monkeypatch, nk):
    m = gfk.Medium(gfk.Stack(gfk.Layer(*t) for t in SOIL), formulation=gfk.DUNKIN, omega_imag=0.8, engine=engine)
    freqs, ranges = np.array([7.0, 31.0, 120.0, 260.0]), np.linspace(1.0, 21.0, 9)
    want, ost = oracle.bank_spectra(SOIL, ranges, freqs, samples=nk, kmax=40.0, formulation=oracle.DUNKIN, omega_imag=0.8)
    assert (ost == 0).all()
    for variant in ("0", "4", "10"):
        monkeypatch.setenv("GFK_PROP_VARIANT", variant)
        got, status = m.bank_spectra(ranges, freqs, gfk.Integration(nk, 0.0, 40.0))
        assert (status == 0).all()
        assert max(rel_l2(g, w) for g, w in zip(got, want)) < 1e-9

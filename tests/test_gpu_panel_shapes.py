"""Panels in every kind of block against the CPU oracle, on the soils and at the wavenumber
counts of test_gpu_panels and to its tolerance. A forced launch shape takes panels at any
size: 64, 128 and 256 threads (half a panel, one and two at once where every
wavenumber of a refused one is solved), all nodes at once, one item per block and persistent;
the sum fused in for 1 and 5 ranges. One bank is large enough for panels unforced."""
import numpy as np
import pytest

from conftest import rel_l2
from test_gpu_panels import SOILS

pytestmark = pytest.mark.gpu


def medium(gfk, engine, soil):
    st, wi = SOILS[soil]
    return st, wi, gfk.Medium(gfk.Stack(gfk.Layer(*t) for t in st), formulation=gfk.DUNKIN, omega_imag=wi, engine=engine)


@pytest.mark.parametrize("nk", [64, 96, 97, 160, 161, 512, 1024, 1056, 1057, 3001])
@pytest.mark.parametrize("soil", SOILS)
def test_panel_shapes_against_oracle(gfk, engine, oracle, monkeypatch, soil, nk):
    st, wi, m = medium(gfk, engine, soil)
    freqs = np.array([7.0, 31.0, 120.0, 260.0])
    shapes = [gfk.prop_shape(v) for v in range(11)]
    assert {s["threads"] for s in shapes} == {64, 128, 256} and {s["persistent"] for s in shapes} == {False, True}
    for nr in (1, 5, 9):
        ranges = np.linspace(1.0, 21.0, nr)
        want, ost = oracle.bank_spectra(st, ranges, freqs, samples=nk, kmax=40.0, formulation=oracle.DUNKIN,
                                        omega_imag=wi)
        assert (ost == 0).all()
        for s in shapes if nr == 9 else shapes[:1]:  # the fused sum has one shape of panels
            monkeypatch.setenv("GFK_PROP_VARIANT", str(s["index"]))
            got, status = m.bank_spectra(ranges, freqs, gfk.Integration(nk, 0.0, 40.0))
            assert (status == 0).all()
            worst = max(rel_l2(g, w) for g, w in zip(got, want))
            assert worst < 1e-9, (s, nr, worst)


@pytest.mark.parametrize("soil", ["low_loss", "heavy_plate"])
def test_unforced_panels_against_oracle(gfk, engine, oracle, soil):
    st, wi, m = medium(gfk, engine, soil)
    freqs, ranges, nk = np.linspace(4.0, 300.0, 80), np.linspace(1.0, 21.0, 9), 12001
    p = gfk.Plan(m, ranges, freqs, gfk.Integration(nk, 0.0, 40.0), engine=engine)
    p.execute()
    assert p.prop_shape()["index"] < 64
    got, status = p.download()
    p.close()
    assert (status == 0).all()
    want, ost = oracle.bank_spectra(st, ranges, freqs, samples=nk, kmax=40.0, formulation=oracle.DUNKIN, omega_imag=wi)
    assert (ost == 0).all()
    assert max(rel_l2(g, w) for g, w in zip(got, want)) < 1e-9

"""Panels of the integrand from Chebyshev nodes (gfk_panel.cuh) against the CPU
oracle, which solves every wavenumber: FP64 Dunkin path, rel-L2 <= 1e-9 per
frequency, as in test_gpu_parity. Wavenumber counts put the last panel on both
sides of the shortest one that is tried (33 wavenumbers) and of a work item;
nr = 1 and 5 take the sum fused into the propagator (node weights), 9 the GEMM."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

SOILS = {
    "graded": ([(0.8, 240.0, 120.0, 1600.0, 10.0, 20.0), (0.8, 480.0, 240.0, 1750.0, 30.0, 60.0),
                (0.8, 800.0, 400.0, 1900.0, 45.0, 90.0), (0.0, 1200.0, 600.0, 2100.0, 60.0, 120.0)], 0.8),
    # poles far narrower than a panel's node spacing: the tails must refuse them
    "low_loss": ([(1.3, 300.0, 150.0, 1700.0, 1e5, 2e5), (0.0, 900.0, 450.0, 2000.0, 1e5, 2e5)], 0.0),
    # a heavy stiff plate on light soil: its flexural wave is slower than every layer's Rayleigh wave
    "heavy_plate": ([(0.3, 500.0, 250.0, 9000.0, 50.0, 100.0), (0.0, 500.0, 250.0, 600.0, 40.0, 80.0)], 0.5),
}


@pytest.mark.parametrize("nk", [64, 96, 97, 160, 161, 512, 1024, 1056, 1057, 3001])
@pytest.mark.parametrize("soil", SOILS)
def test_panels_against_oracle(gfk, engine, oracle, soil, nk):
    st, wi = SOILS[soil]
    m = gfk.Medium(gfk.Stack(gfk.Layer(*t) for t in st), formulation=gfk.DUNKIN, omega_imag=wi, engine=engine)
    freqs = np.array([7.0, 31.0, 120.0, 260.0])
    opt = gfk.Integration(nk, 0.0, 40.0)
    for nr in (1, 5, 9):
        ranges = np.linspace(1.0, 21.0, nr)
        got, status = m.bank_spectra(ranges, freqs, opt)
        assert (status == 0).all()
        want, ost = oracle.bank_spectra(st, ranges, freqs, samples=nk, kmax=40.0, formulation=oracle.DUNKIN,
                                        omega_imag=wi)
        assert (ost == 0).all()
        worst = max(rel_l2(g, w) for g, w in zip(got, want))
        assert worst < 1e-9, worst


def test_panels_on_per_frequency_grids(gfk, engine, oracle):
    """The row path's panels: items that end inside the row, k u without the static term."""
    st, wi = SOILS["graded"]
    m = gfk.Medium(gfk.Stack(gfk.Layer(*t) for t in st), formulation=gfk.DUNKIN, omega_imag=wi, engine=engine)
    freqs = np.array([3.0, 17.0, 111.0])
    ranges = np.array([0.6, 4.0, 23.0])
    got, status = m.bank_spectra(ranges, freqs)
    assert (status == 0).all()
    want, ost = oracle.bank_spectra(st, ranges, freqs, formulation=oracle.DUNKIN, omega_imag=wi)
    assert max(rel_l2(g, w) for g, w in zip(got, want)) < 1e-9

"""Per-frequency grids (the row sums over items of wavenumbers, J0 in the
loop) against the CPU oracle. FP64 Dunkin path: rel-L2 <= 1e-9, as in
test_gpu_parity."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr", [1, 2, 3, 8, 9, 17])
def test_row_sums_against_oracle(gfk, engine, oracle, nr):
    """Range tiles of 1, 2, 4 and 8 full and ragged; rows from one item (a few
    thousand wavenumbers) to hundreds (131k, whose step the low frequency sets);
    arguments k r on both sides of the asymptotic form's start."""
    st = [(1.5, 420.0, 180.0, 1650.0, 20.0, 40.0), (0.0, 800.0, 350.0, 2000.0, 25.0, 50.0)]
    m = gfk.Medium(gfk.Stack(gfk.Layer(*t) for t in st), formulation=gfk.DUNKIN, engine=engine)
    ranges = np.geomspace(0.7, 33.0, nr)
    freqs = np.array([2.0, 21.0, 77.7, 140.0])
    got, status = m.bank_spectra(ranges, freqs)
    assert (status == 0).all()
    want, ost = oracle.bank_spectra(st, ranges, freqs, formulation=oracle.DUNKIN)
    assert (ost == 0).all()
    assert max(rel_l2(g, w) for g, w in zip(got, want)) < 1e-9
    # one frequency on its own: other item sizes, the same sums to rounding
    one = m.vertical_displacement_multi(ranges, freqs[1])
    assert rel_l2(one, want[1]) < 1e-9

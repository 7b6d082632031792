"""Impulse responses on both sides of the query count from which a block has only
the transform's threads (592): each query's response bit for bit that of a short call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 16, 128, 256, 512, 1024, 4096])
def test_response_does_not_depend_on_the_count(gfk, engine, n):
    rng = np.random.default_rng(n)
    bins, count = n // 2 + 1, 5
    data = rng.normal(size=(count, bins, 2)).astype(np.float32)
    h = gfk.Header(gfk.Provenance("x"), gfk.uniform(500.0, 200.0, 1700.0, 25.0), 800.0, n, gfk.RangeGrid(1.0, 9.0, count),
                   "vertical_displacement", "m/N")
    bank = gfk.Bank(h, data)
    ranges = np.linspace(1.0, 9.0, 593)
    length = max(1, n - 1)
    whole = bank.impulse_responses(ranges, length, engine=engine)
    assert whole.shape == (593, length)
    assert np.array_equal(bank.impulse_responses(ranges[:592], length, engine=engine), whole[:592])
    assert np.array_equal(bank.impulse_responses(ranges[-7:], length, engine=engine), whole[-7:])

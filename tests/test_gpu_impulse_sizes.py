"""Impulse responses at every transform size (2 to 4096: each first radix, one
to four passes, blocks from one warp) and at odd and even lengths, against the
numpy restatement: the tolerance of test_gpu_consume, 1e-12 of the largest
sample."""
import pathlib
import sys

import numpy as np
import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT / "oracle"))
import bank_oracle as BO  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2 ** e for e in range(1, 13)])
def test_every_transform_size(gfk, engine, n):
    rng = np.random.default_rng(n)
    bins, count, fs = n // 2 + 1, 3, 800.0
    data = (rng.normal(size=(count, bins, 2)) * np.exp(-0.01 * np.arange(bins))[None, :, None]).astype(np.float32)
    data[1, bins // 2] = 0.0  # an exact zero answers zero in the brackets that touch it
    h = gfk.Header(gfk.Provenance("x"), gfk.uniform(500.0, 200.0, 1700.0, 25.0), fs, n, gfk.RangeGrid(1.0, 5.0, count),
                   "vertical_displacement", "m/N")
    bank = gfk.Bank(h, data)
    ranges = np.array([1.0, 1.7, 3.0, 4.2, 5.0])
    sensor = rng.normal(size=bins) + 1j * rng.normal(size=bins)
    for length in sorted({1, max(1, n // 4), max(1, n // 2 - 1), n - 1, n}):
        want = BO.impulse_responses(data, (1.0, 5.0), fs, n, ranges, length, sensor=sensor)
        got = bank.impulse_responses(ranges, length, sensor=sensor, engine=engine)
        assert got.shape == want.shape
        assert np.abs(got - want).max() <= 1e-12 * max(np.abs(want).max(), 1e-300), length

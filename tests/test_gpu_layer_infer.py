"""The inference layers' persistent kernel over several blocks of rows per SM
pair (37 pairs a slab, 256 rows a block, two accumulators in turn): a row's answer is
the one it gets alone, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 9472 rows, the last count with a tile per CTA, then pairs: a second block for one pair, a
# last block of 128 rows, 236 blocks; each against 256 to 1024 rows, a tile per CTA
@pytest.mark.parametrize("ns,nf,nr", [(37, 256, 1), (37, 257, 1), (37, 769, 1), (59, 512, 2)])
def test_rows_do_not_depend_on_their_block(gfk, engine, ns, nf, nr):
    net = gfk.surrogate.Net(gfk.surrogate.NetConfig(batch=128, seed=12), engine)
    try:
        net.set_scales(1.0, 64.0, 0.9765625, 500.0, (-22.0, 2.5, 0.0045, 0.0005))
        p = gfk.surrogate.draw(ns, 6)
        freqs = np.linspace(1.0, 480.0, nf)
        ranges = np.linspace(2.0, 60.0, nr)
        whole = net.predict(p, ranges, freqs)
        assert whole.shape == (ns, nf, nr) and np.isfinite(whole).all()
        for s in range(0, ns, 4):  # every fourth soil by itself: nf * nr rows
            assert (net.predict(p[s:s + 1], ranges, freqs)[0] == whole[s]).all()
    finally:
        net.close()

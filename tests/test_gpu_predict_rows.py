"""The network's rows at ragged counts: a row's answer does not depend on where
in a call it lies (warps of 32 rows, blocks of 64 and 256, GEMM tiles of 128), bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def net(gfk, engine):
    n = gfk.surrogate.Net(gfk.surrogate.NetConfig(batch=128, seed=11), engine)
    n.set_scales(1.0, 64.0, 0.9765625, 500.0, (-22.0, 2.5, 0.0045, 0.0005))
    yield n
    n.close()


@pytest.mark.parametrize("ns,nf,nr", [(1, 1, 1), (1, 31, 1), (3, 11, 1), (1, 64, 1), (5, 13, 3), (2, 129, 1), (9, 57, 2)])
def test_rows_do_not_depend_on_their_place(gfk, net, ns, nf, nr):
    p = gfk.surrogate.draw(ns, 5)
    freqs = np.linspace(1.0, 480.0, nf)
    ranges = np.linspace(2.0, 60.0, nr)
    whole = net.predict(p, ranges, freqs)
    assert whole.shape == (ns, nf, nr) and np.isfinite(whole).all()
    for s in (0, ns - 1):
        for f in (0, nf // 2, nf - 1):
            for r in (0, nr - 1):
                one = net.predict(p[s:s + 1], ranges[r:r + 1], freqs[f:f + 1])
                assert one[0, 0, 0] == whole[s, f, r]

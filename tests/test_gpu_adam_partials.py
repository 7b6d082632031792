"""AdamW's gradient sums and weight copies at the batch sizes where the split of
the work changes (the head has one partial per 32 samples: one thread a
parameter up to 32, a block for 32 parameters, 128 partials at a time, above)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HEAD = 2 * 512 + 2


@pytest.fixture(scope="module")
def one_cell(gfk, engine):
    """A data set of one soil, range and frequency: every sample is the same, so
    the mean gradient does not depend on the batch size."""
    ds = gfk.surrogate.Dataset(gfk.surrogate.draw(1, 3), gfk.surrogate.LabelGrid(
        ranges=np.array([5.0]), fs=60.0, n=2, nk=1024), engine=engine).fill(batch_soils=1)
    yield ds
    ds.close()


def first_step(gfk, engine, ds, batch):
    sur = gfk.surrogate
    # one step at rate 1 with eps = 1 moves a parameter by g / (|g| + 1)
    net = sur.Net(sur.NetConfig(batch=batch, warmup_steps=1, total_steps=10, lr_max=1.0, eps=1.0, seed=7,
                                loss_mode=gfk._native.LOSS_PLAIN), engine)
    net.set_scales(1.0, 64.0, 1.0, 500.0, [-20.0, 2.5, 0.0, 1.0])
    before = net.params()
    net.train(ds, [0], 1)
    return net, before, net.params()


@pytest.mark.parametrize("batch", [128, 1152, 4096, 4224, 8192])
def test_head_gradient_and_weight_copies(gfk, engine, one_cell, batch):
    step = []
    for b in (1024, batch):
        net, p0, p1 = first_step(gfk, engine, one_cell, b)
        u = (p0.astype(np.float64) - p1)[-HEAD:]
        step.append(u / (1.0 - np.abs(u)))
        if b == batch:
            # the copies W and W^T that the step wrote are those of its parameters
            rng = np.random.default_rng(1)
            X = rng.uniform(-1, 1, (batch, 128)).astype(np.float32)
            Y = rng.normal(size=(batch, 2)).astype(np.float32)
            g0, l0 = net.probe(X, Y)
            net.set_params(p1)
            g1, l1 = net.probe(X, Y)
            assert (g0 == g1).all() and (l0 == l1).all()
        net.close()
    # 4 + 8 + 264 additions of one sign in FP32 on each side, and the parameter's own rounding
    tol = 2 * 276 * 2.0 ** -24 * np.abs(step[0]) + 2.0 ** -22 * max(1.0, np.abs(p1[-HEAD:]).max())
    assert np.abs(step[0]).max() > 1e-3
    assert (np.abs(step[1] - step[0]) <= tol).all()

"""Which plans share a tuned propagator shape: those of as many layers and wavenumbers, the
same kind of sum, and few or many items of 1024 wavenumbers (2500 in the window) alike."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_shape_is_timed_per_size_and_sum(gfk):
    eng = gfk.Engine(0)
    stack = gfk.Stack([gfk.Layer(0.8, 240.0, 120.0, 1600.0, 10.0, 20.0), gfk.Layer(0.0, 1200.0, 600.0, 2100.0, 60.0, 120.0)])

    def timed(nf, nk, quadrature):
        m = gfk.Medium(stack, formulation=gfk.DUNKIN, omega_imag=0.8, engine=eng, quadrature=quadrature)
        p = gfk.Plan(m, np.linspace(1.0, 21.0, 9), np.linspace(5.0, 240.0, nf), gfk.Integration(nk, 0.0, 40.0), engine=eng)
        p.execute()
        n = len(p.tuning()[1])
        p.close()
        return n

    plain, split = gfk.PLAIN_FP64, gfk.SPLIT_INT8
    shapes = timed(320, 3001, plain)  # 960 items
    assert shapes > 1
    assert timed(833, 3001, plain) == 0       # 2499: few as well
    assert timed(834, 3001, plain) == shapes  # 2502: many
    assert timed(320, 3001, plain) == 0 and timed(2000, 3001, plain) == 0
    assert timed(320, 3001, split) == shapes and timed(833, 3001, split) == 0
    assert timed(2000, 3001, split) == shapes
    assert timed(320, 3002, plain) == shapes
    eng.close()

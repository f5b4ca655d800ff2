"""Launch shapes timed for an adjoint window (its launches store the moments of
every step) stay the window's: plain steps afterwards take what plain steps
were timed for, as on a handle of the same kind that had no window."""
import numpy as np
import pytest

import lagrangianrbnudging_b200 as lb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("store", [0, 1])
def test_plain_steps_after_a_window(precision, store):
    nx, ny = 520, 250 + store  # (a kind of its own: nothing timed before)
    kw = dict(lb.closure(nx, ny, Ra=1e6, Pr=1.0, U=0.1), precision=precision)
    rng = np.random.default_rng(1)
    steps = np.arange(5, 21, 5, dtype=np.int32)
    x, y = rng.uniform(1, nx - 1, (4, 50)), rng.uniform(2, ny - 1, (4, 50))
    T0 = 0.5 - (np.arange(ny) + 0.5)[:, None] / ny + 0.01 * rng.standard_normal((ny, nx))
    with lb.Run(**kw) as a, lb.Run(**kw) as b:
        a.init_conduction(3, 5e-2)
        a.step(30)
        b.adjoint_set_store(store)
        b.adjoint_set_obs(steps, x, y, 0.1 * rng.standard_normal((4, 50)))
        J, grad = b.adjoint_window(T0, 20, 8)
        first = b.pair_shape()["shape"]
        b.init_conduction(3, 5e-2)
        b.step(30)
        assert b.pair_shape() == a.pair_shape()
        assert first >= 0 or a.pair_shape()["shape"] >= 0
        for p, q in zip(a.get_populations(), b.get_populations()):
            np.testing.assert_array_equal(p, q)
        # the window again, on either's shapes
        for r in (a, b):
            r.adjoint_set_store(store)
            r.adjoint_set_obs(steps, x, y, np.zeros((4, 50)))
        (Ja, ga), (Jb, gb) = a.adjoint_window(T0, 20, 8), b.adjoint_window(T0, 20, 8)
        assert Ja == Jb
        np.testing.assert_array_equal(ga, gb)

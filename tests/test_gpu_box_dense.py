"""Box nudging with many observations in a cell (csrc/nudge_kernels.cu, chains
of contributions): bit-identical to the oracle around the lengths at which a
cell's slots and chains fill, and a step's time in proportion to the
observations at a given density."""
import numpy as np
import pytest

import lagrangianrbnudging_b200 as lb
from tests.test_gpu_box_cells import box_case, test_cells_match_the_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,spread,drift", [(10, 0.0, 3.0), (23, 0.0, 3.0), (24, 0.0, 3.0), (25, 0.0, 3.0), (41, 0.0, 9.0),
                                            (3000, 40.0, 2.0)])
def test_chains_match_the_oracle(n, spread, drift):
    test_cells_match_the_oracle(n, spread, drift)


def seconds_per_step(nx, ny, n, nt=10):
    import torch

    rng = np.random.default_rng(1)
    x, y = rng.uniform(1, nx - 1, n), rng.uniform(2, ny - 1, n)
    T, ids = rng.uniform(-0.5, 0.5, n), np.arange(n, dtype=np.int32)
    with lb.Run(**lb.closure(nx, ny, Ra=1e6, Pr=1.0, U=0.1), precision="fp64", twall="adiabatic", nudge="refbox",
                alpha=0.5, ntempread=nt, nobs=n) as r:
        r.init_conduction(3, 1e-2)
        r.nudge_init(x, y, T, ids)
        s = torch.cuda.Stream()
        r.set_stream(s.cuda_stream)
        best = 1e30
        for _ in range(4):
            r.nudge_load(x, y, ids, T)
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(s)
            r.step(nt)
            b.record(s)
            r.sync()
            best = min(best, a.elapsed_time(b) * 1e-3 / nt)
        r.set_stream(None)
    return best


def test_time_goes_with_the_observations():
    """16 times the nodes and the observations: 16 times the work at most (of
    which a small grid hides some in launches), not 256 times"""
    small, large = seconds_per_step(256, 128, 1 << 14), seconds_per_step(1024, 512, 1 << 18)
    assert large < 32 * small, (small, large)

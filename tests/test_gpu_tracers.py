"""Runs whose particles are all tracers take the particle kernels without the
derivative stencil, and ride in the fused launches, whatever beta is: equal to
single steps bit for bit, and again after inertial particles take their places."""
import numpy as np
import pytest

import lagrangianrbnudging_b200 as lb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("full", [0, 1])
def test_tracers_with_beta(precision, full):
    nx, ny, n = 128, 64, 300
    rng = np.random.default_rng(3)
    x, y = rng.uniform(0.5, nx, n), rng.uniform(1.0, ny, n)
    z, ids = np.zeros(n), np.arange(n, dtype=np.int32)
    runs = []
    for pairs in (0, 1):
        r = lb.Run(**lb.closure(nx, ny, Ra=1e5, Pr=1.0, U=0.1), precision=precision, nprtcl=n, noutconfig=3,
                   record_slots=32, beta=0.4, record_full=full)
        r.set_graph(0)
        r.set_pairs(pairs)
        if pairs:
            r.set_pair_shape(7)
        r.init_conduction(7, 5e-2)
        runs.append(r)
    for kinds in (np.zeros(n, np.int32), (np.arange(n) % 2).astype(np.int32), np.zeros(n, np.int32)):
        out = []
        for r in runs:
            r.set_particles(ids, x, y, z, z, kinds, np.where(kinds == 1, 0.05, 0.0))
            r.step(21)
            out.append((r.get_particles(), r.drain_records_array()))
        (pa, ra), (pb, rb) = out
        for k in pa:
            np.testing.assert_array_equal(pb[k], pa[k], err_msg=k)
        np.testing.assert_array_equal(rb[0], ra[0])
        np.testing.assert_array_equal(rb[1], ra[1])
    for r in runs:
        r.close()

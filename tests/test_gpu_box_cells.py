"""Box nudging's cell lists (csrc/nudge_kernels.cu): bit-identical to the
oracle where the lists can go wrong -- one observation, cells within their own
slots, cells over them, cells that are touched in one step and not in the
next (cleared), boxes over the periodic edge and at the walls."""
import numpy as np
import pytest

import lagrangianrbnudging_b200 as lb
from tests.golden import cases

pytestmark = pytest.mark.gpu


def box_case(n, spread, drift, nx=72, ny=41, nt=4, nsteps=16, seed=3):
    rng = np.random.default_rng(seed)
    base = lb.closure(nx, ny, Ra=1e5, Pr=1.0, U=0.1)
    x = (nx - 2 + rng.uniform(-spread, spread, n)) % nx
    y = np.clip(6.0 + rng.uniform(-spread, spread, n), 1.0, ny)
    T = rng.uniform(-0.5, 0.5, n)
    ids = (rng.permutation(n) + 7).astype(np.int32)
    init = dict(x=x.copy(), y=y.copy(), T=T.copy(), id=ids)
    files = {}
    for s in range(nt, nsteps + nt, nt):
        x = (x + drift + rng.normal(0, 0.5, n)) % nx
        y = np.clip(y + 0.7 * drift + rng.normal(0, 0.5, n), 1.0, ny)
        p = rng.permutation(n)
        files[s] = dict(x=x[p].copy(), y=y[p].copy(), id=ids[p].copy(), temp=T[p].copy())
    j = np.arange(ny)
    Tic = (0.5 - (j + 0.5) / ny)[:, None] + 1e-2 * rng.uniform(-1, 1, (ny, nx))
    params = dict(base, twall="adiabatic", nudge="refbox", alpha=0.2, ntempread=nt)
    return dict(nx=nx, ny=ny, nprtcl=n, nsteps=nsteps, ntempread=nt, alpha=0.2, base=base, params=params, Tic=Tic,
                init_obs=init, files=files)


@pytest.mark.parametrize("n,spread,drift", [(1, 0.0, 9.0), (8, 1.0, 3.0), (9, 1.0, 0.1), (40, 30.0, 5.0), (300, 4.0, 2.0)])
def test_cells_match_the_oracle(n, spread, drift):
    c = box_case(n, spread, drift)
    want = cases.run_oracle_nudge(c)
    st = cases.nudge_initial_state(c)
    io = c["init_obs"]
    with lb.Run(**c["base"], precision="fp64", twall="adiabatic", nudge="refbox", alpha=c["alpha"],
                ntempread=c["ntempread"], nobs=n) as r:
        r.set_populations(st["f"], st["g"])
        r.set_moments(st["rho"], st["u"], st["v"], st["T"])
        r.nudge_init(io["x"], io["y"], io["T"], io["id"])
        for s in range(1, c["nsteps"] + 1):
            if s % c["ntempread"] == 1:
                d = c["files"][s + c["ntempread"] - 1]
                r.nudge_load(d["x"], d["y"], d["id"], d["temp"])
            r.step(1)
        r.sync()
        f, g = r.get_populations()
        m = r.get_moments()
    np.testing.assert_array_equal(f, want["f"])
    np.testing.assert_array_equal(g, want["g"])
    for k in ("T", "u", "v"):
        np.testing.assert_array_equal(m[k], want[k], err_msg=k)

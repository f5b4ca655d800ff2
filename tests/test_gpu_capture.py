"""Graphs that a caller captures from lbrb_step, replayed: as many steps taken
directly give the same state bit for bit."""
import numpy as np
import pytest

import lagrangianrbnudging_b200 as lb
from tests.golden import cases
from tests.test_gpu_box_cells import box_case

pytestmark = pytest.mark.gpu


def capture(r, s, n):
    """a graph of r.step(n) on stream s (which r is on)"""
    import torch

    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s, capture_error_mode="thread_local"):
        r.step(n)
    return g


@pytest.mark.parametrize("nt", [4, 6])
def test_box_nudged_interval(nt):
    """a captured interval between two observation files, replayed with each
    file: interval lengths that are a multiple of the three sets of cell lists
    and that are not; cells touched in one step and not in the next"""
    import torch

    c = box_case(40, 30.0, 5.0, nt=nt, nsteps=5 * nt)
    st = cases.nudge_initial_state(c)
    io = c["init_obs"]

    def run():
        r = lb.Run(**c["base"], precision="fp64", twall="adiabatic", nudge="refbox", alpha=c["alpha"],
                   ntempread=nt, nobs=c["nprtcl"])
        r.set_populations(st["f"], st["g"])
        r.set_moments(st["rho"], st["u"], st["v"], st["T"])
        r.nudge_init(io["x"], io["y"], io["T"], io["id"])
        return r

    def load(r, s):
        d = c["files"][s]
        r.nudge_load(d["x"], d["y"], d["id"], d["temp"])

    with run() as a, run() as b:
        for s in range(nt, c["nsteps"] + 1, nt):
            load(b, s)
            b.step(nt)
        stream = torch.cuda.Stream()
        a.set_stream(stream.cuda_stream)
        load(a, nt)
        a.step(nt)
        load(a, 2 * nt)
        g = capture(a, stream, nt)
        g.replay()
        for s in range(3 * nt, c["nsteps"] + 1, nt):
            torch.cuda.synchronize()
            load(a, s)
            g.replay()
        torch.cuda.synchronize()
        a.set_stream(None)
        for p, q in zip(a.get_populations(), b.get_populations()):
            np.testing.assert_array_equal(p, q)
        ma, mb = a.get_moments(), b.get_moments()
        for k in ma:
            np.testing.assert_array_equal(ma[k], mb[k], err_msg=k)
        del g

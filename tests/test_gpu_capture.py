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


def free_run(precision, nx, ny, kind, rows=0):
    """kind: no particles, few tracers, or few inertial particles (d/dt reads
    the u, v of the step before); rows: of a repeating series of observations"""
    n = 0 if kind == "none" else 96
    kw = dict(nudge="bilinear", alpha=0.2, nobs=40, obs_cycle=1) if rows else {}
    r = lb.Run(**lb.closure(nx, ny, Ra=1e6, Pr=1.0, U=0.1), precision=precision, nprtcl=n,
               beta=0.5 if kind == "inertial" else 0.0, **kw)
    r.set_pairs(1)
    if rows:
        rng = np.random.default_rng(3)
        r.nudge_obs(1, rng.uniform(0, nx, (rows, 40)), rng.uniform(1, ny, (rows, 40)), rng.uniform(-0.5, 0.5, (rows, 40)))
    r.init_conduction(11, 5e-2)
    if n:
        rng = np.random.default_rng(5)
        ptype = np.full(n, 1 if kind == "inertial" else 0, np.int32)
        z = np.zeros(n)
        r.set_particles(np.arange(n, dtype=np.int32), rng.uniform(0.5, nx + 0.5, n), rng.uniform(1.0, ny, n), z, z,
                        ptype, np.where(ptype == 1, 1.0 / 50.0, 0.0))
    return r


def assert_same(a, b):
    for p, q in zip(a.get_populations(), b.get_populations()):
        np.testing.assert_array_equal(p, q)
    ma, mb = a.get_moments(), b.get_moments()
    for k in ma:
        np.testing.assert_array_equal(ma[k], mb[k], err_msg=k)
    if a.np:
        pa, pb = a.get_particles(), b.get_particles()
        for k in pa:
            np.testing.assert_array_equal(pa[k], pb[k], err_msg=k)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("nx,ny", [(128, 64), (2048, 1024)])
@pytest.mark.parametrize("kind,n,between", [("none", 8, 0), ("none", 24, 0), ("tracers", 12, 12), ("inertial", 12, 12),
                                            ("inertial", 24, 36)])
def test_replays_after_tuned_calls(precision, nx, ny, kind, n, between):
    """a call captured once its launch shapes are timed, whichever they are,
    over lengths that end in the buffers they started from; with particles
    also around direct calls of such lengths"""
    import torch

    with free_run(precision, nx, ny, kind) as a, free_run(precision, nx, ny, kind) as b:
        stream = torch.cuda.Stream()
        a.set_stream(stream.cuda_stream)
        a.step(21)
        g = capture(a, stream, n)
        total = 21
        for q in range(4):
            with torch.cuda.stream(stream):
                g.replay()
            total += n
            if between and q % 2:
                a.step(between)
                total += between
        torch.cuda.synchronize()
        a.set_stream(None)
        b.set_pairs(0)
        b.step(total)
        assert_same(a, b)
        del g


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("kind", ["none", "inertial"])
@pytest.mark.parametrize("n", [6, 18])
@pytest.mark.parametrize("pairs", [0, 1])
def test_nudged_replays(precision, kind, n, pairs):
    """bilinear nudging toward a series that repeats every captured call"""
    import torch

    nx, ny = 128, 64
    with free_run(precision, nx, ny, kind, rows=6) as a, free_run(precision, nx, ny, kind, rows=6) as b:
        a.set_pairs(pairs)
        stream = torch.cuda.Stream()
        a.set_stream(stream.cuda_stream)
        a.step(24)
        g = capture(a, stream, n)
        with torch.cuda.stream(stream):
            for _ in range(3):
                g.replay()
        torch.cuda.synchronize()
        a.set_stream(None)
        b.set_pairs(0)
        b.step(24 + 3 * n)
        assert_same(a, b)
        del g

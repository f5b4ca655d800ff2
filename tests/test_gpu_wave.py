"""The FP32 strip kernels (csrc/lb_pair.cuh: wave_march), one warp per strip:
bit-identical to single steps where their index arithmetic can go wrong --
grids narrower than a strip, one strip, just over one, widths not a multiple
of a strip or of 32, the smallest heights, chunks of one row and of many."""
import numpy as np
import pytest

import lagrangianrbnudging_b200 as lb

pytestmark = pytest.mark.gpu


def make(nx, ny, pairs, shape, nprtcl=0, nobs=0, seed=5):
    kw = dict(lb.closure(nx, ny, Ra=1e5, Pr=1.0, U=0.05), precision="fp32", nprtcl=nprtcl,
              noutconfig=3 if nprtcl else 0, record_slots=64, beta=0.5, record_full=1)
    if nobs:
        kw.update(nudge="bilinear", alpha=0.2, nobs=nobs, obs_cycle=1)
    r = lb.Run(**kw)
    r.set_graph(0)
    r.set_pairs(pairs)
    if pairs and shape >= 0:
        r.set_pair_shape(shape)
    r.init_conduction(seed, 5e-2)
    rng = np.random.default_rng(seed)
    if nprtcl:
        ptype = (np.arange(nprtcl) % 2).astype(np.int32)
        z = np.zeros(nprtcl)
        r.set_particles(np.arange(nprtcl, dtype=np.int32), rng.uniform(0.5, nx, nprtcl), rng.uniform(1.0, ny, nprtcl),
                        z, z, ptype, np.where(ptype == 1, 0.05, 0.0))
    if nobs:
        r.nudge_obs(1, rng.uniform(0.0, nx, (5, nobs)), rng.uniform(1.0, ny, (5, nobs)), rng.uniform(-0.5, 0.5, (5, nobs)))
    return r


def state(r):
    f, g = r.get_populations()
    out = dict(f=f, g=g, **r.get_moments())
    if r.np:
        out.update({"p" + k: v for k, v in r.get_particles().items()})
        out["steps"], out["rec"] = r.drain_records_array()
    return out


def same(a, b, calls):
    for n in calls:
        a.step(n)
        b.step(n)
        sa, sb = state(a), state(b)
        for k in sa:
            np.testing.assert_array_equal(sb[k], sa[k], err_msg=f"{k} after a call of {n} steps")


@pytest.mark.parametrize("nx", [4, 8, 56, 60, 64, 112, 116, 120, 124, 484])
@pytest.mark.parametrize("ny", [3, 4, 7, 90])
@pytest.mark.parametrize("shape", [9, 14])
def test_strip_edges(nx, ny, shape):
    with make(nx, ny, 0, -1) as a, make(nx, ny, 1, shape) as b:
        same(a, b, (2, 3, 13))


@pytest.mark.parametrize("nx,ny", [(64, 5), (180, 61)])
def test_strip_edges_with_particles_and_nudging(nx, ny):
    with make(nx, ny, 0, -1, 30, 40) as a, make(nx, ny, 1, 12, 30, 40) as b:
        same(a, b, (2, 3, 12))


@pytest.mark.parametrize("nx,ny", [(4, 5), (56, 3), (60, 8), (64, 33), (232, 700), (512, 256)])
@pytest.mark.parametrize("nprtcl,every", [(0, 0), (30, 2), (30, 5)])
def test_four_steps_per_launch(nx, ny, nprtcl, every):
    """automatic launches (four, two and one steps, whichever the tuner
    keeps) against single steps: calls around multiples of four, records on
    every step of a group (every = 2: two in a group, so pairs)"""
    def run(pairs):
        kw = dict(lb.closure(nx, ny, Ra=1e5, Pr=1.0, U=0.05), precision="fp32", nprtcl=nprtcl, noutconfig=every,
                  record_slots=64, beta=0.5, record_full=1)
        r = lb.Run(**kw)
        r.set_graph(0)
        r.set_pairs(pairs)
        r.init_conduction(7, 5e-2)
        if nprtcl:
            rng = np.random.default_rng(7)
            ptype = (np.arange(nprtcl) % 2).astype(np.int32)
            z = np.zeros(nprtcl)
            r.set_particles(np.arange(nprtcl, dtype=np.int32), rng.uniform(0.5, nx, nprtcl),
                            rng.uniform(1.0, ny, nprtcl), z, z, ptype, np.where(ptype == 1, 0.05, 0.0))
        return r

    with run(0) as a, run(1) as b:
        same(a, b, (5, 6, 7, 8, 9, 23))

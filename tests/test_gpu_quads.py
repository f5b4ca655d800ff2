"""The four-step kernel (csrc/lb_kernels.cu: lb_wave4_kernel), forced:
bit-identical to single steps where its index arithmetic can go wrong -- grids
narrower than a strip of 56 columns, one strip, just over one, widths that are
no multiple of a strip, the smallest heights, chunks of one row, of a few and
of many -- in every launch shape, with records at each of the four steps."""
import numpy as np
import pytest

import lagrangianrbnudging_b200 as lb

pytestmark = pytest.mark.gpu


def make(precision, nx, ny, shape, nprtcl=0, every=0, beta=0.5):
    r = lb.Run(**lb.closure(nx, ny, Ra=1e5, Pr=1.0, U=0.05), precision=precision, nprtcl=nprtcl, noutconfig=every,
               record_slots=64, beta=beta, record_full=1 if beta else 0)
    r.set_graph(0)
    r.set_pairs(0 if shape is None else 1)
    if shape is not None:
        r.set_pair_shape(0)
        r.set_quad_shape(shape)
    r.init_conduction(7, 5e-2)
    if nprtcl:
        rng = np.random.default_rng(7)
        ptype = (np.arange(nprtcl) % 2).astype(np.int32)
        z = np.zeros(nprtcl)
        r.set_particles(np.arange(nprtcl, dtype=np.int32), rng.uniform(0.5, nx, nprtcl), rng.uniform(1.0, ny, nprtcl),
                        z, z, ptype, np.where(ptype == 1, 0.05, 0.0))
    return r


def state(r):
    f, g = r.get_populations()
    out = dict(f=f, g=g, **r.get_moments())
    out["pf"], out["pg"] = r.get_poststream()
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


def assert_launches(r, n, want):
    """n steps take `want` fused launches"""
    r.set_timing(True)
    before = r.get_timing()["lb_step"][1]
    r.step(n)
    assert r.get_timing()["lb_step"][1] - before == want
    r.set_timing(False)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("nx", [4, 8, 52, 56, 60, 64, 112, 116, 484])
@pytest.mark.parametrize("ny", [3, 4, 5, 9, 90])
def test_strip_edges(precision, nx, ny):
    with make(precision, nx, ny, None) as a, make(precision, nx, ny, 0) as b:
        same(a, b, (5, 6, 7, 13))
        assert b.quad_shape() == {"shape": 0, "tuned_ms": 0.0}
        assert_launches(b, 9, 3)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("nx,ny", [(232, 700), (1020, 515), (2048, 1024)])
@pytest.mark.parametrize("shape", range(3))
def test_chunks(precision, nx, ny, shape):
    with make(precision, nx, ny, None) as a, make(precision, nx, ny, shape) as b:
        same(a, b, (9, 22))
        assert_launches(b, 13, 4)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("nx,ny", [(4, 5), (60, 8), (232, 61), (512, 256)])
@pytest.mark.parametrize("every,beta", [(5, 0.5), (5, 0.0), (2, 0.5), (0, 0.5)])
def test_particles_and_records(precision, nx, ny, every, beta):
    """every = 5: a record at each of a group's four steps in turn; every = 2:
    two in each group, which therefore goes in pairs"""
    with make(precision, nx, ny, None, 30, every, beta) as a, make(precision, nx, ny, 1, 30, every, beta) as b:
        same(a, b, (21, 8, 23))
        if every != 2:
            assert_launches(b, 9, 3)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_full_ring_after_four_steps(precision):
    """a call that a full record ring ends where a four-step launch would be
    the last: the state that it leaves, post-stream populations included"""
    nx, ny, n = 116, 40, 30
    runs = []
    for shape in (None, 0):
        r = lb.Run(**lb.closure(nx, ny, Ra=1e5, Pr=1.0, U=0.05), precision=precision, nprtcl=n, noutconfig=8,
                   record_slots=1)
        r.set_graph(0)
        r.set_pairs(0 if shape is None else 1)
        if shape is not None:
            r.set_pair_shape(0)
            r.set_quad_shape(shape)
        r.init_conduction(7, 5e-2)
        rng = np.random.default_rng(7)
        z = np.zeros(n)
        r.set_particles(np.arange(n, dtype=np.int32), rng.uniform(0.5, nx, n), rng.uniform(1.0, ny, n), z, z,
                        np.zeros(n, np.int32), z)
        r.step(3)
        with pytest.raises(lb.LbrbError):
            r.step(30)  # records at 8 and 16; the ring holds one
        runs.append(r)
    a, b = runs
    assert a.istep == b.istep == 15
    for p, q in zip(a.get_poststream() + a.get_populations(), b.get_poststream() + b.get_populations()):
        np.testing.assert_array_equal(q, p)
    for p, q in zip(a.drain_records_array(), b.drain_records_array()):
        np.testing.assert_array_equal(q, p)
    same(a, b, (4, 3))
    for r in runs:
        r.close()


def test_modes():
    assert lb.Run.quad_shapes() == 3
    with make("fp32", 256, 128, -1) as r:
        r.step(30)
        assert r.quad_shape() == {"shape": -1, "tuned_ms": 0.0}
        assert_launches(r, 9, 5)
        r.set_quad_shape(2)
        assert_launches(r, 9, 3)
        r.set_quad_shape(-2)  # (the pair shape is fixed: two steps per launch)
        assert_launches(r, 9, 5)
        for bad in (-3, 3):
            with pytest.raises(lb.LbrbError):
                r.set_quad_shape(bad)
    with lb.Run(**lb.closure(2048, 1024, Ra=1e6, Pr=1.0, U=0.1), precision="fp32") as r:
        r.init_conduction(7, 5e-2)
        r.step(9)
        q = r.quad_shape()
        assert q["shape"] >= -1 and (q["shape"] < 0 or 0 < q["tuned_ms"] < 2 * r.pair_shape()["tuned_ms"])

"""Device memory that a run with particles holds beyond its state: the spare
u, v slots exist only where launches use them, and give way when another
allocation of the handle needs their memory."""
import numpy as np
import pytest

import lagrangianrbnudging_b200 as lb

pytestmark = pytest.mark.gpu

NX, NY = 4096, 2048
PLANE = NX * NY * 4  # bytes of an FP32 field; a u, v slot is two


def run(nprtcl, shape=None, precision="fp32"):
    r = lb.Run(**lb.closure(NX, NY, Ra=1e6, Pr=1.0, U=0.1), precision=precision, nprtcl=nprtcl)
    if shape is not None:
        r.set_pair_shape(shape)
    r.init_conduction(11, 5e-2)
    if nprtcl:
        rng = np.random.default_rng(5)
        z = np.zeros(nprtcl)
        r.set_particles(np.arange(nprtcl, dtype=np.int32), rng.uniform(0.5, NX, nprtcl), rng.uniform(1.0, NY, nprtcl),
                        z, z, np.zeros(nprtcl, np.int32), z)
    return r


def free():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_no_spare_slots_where_nothing_uses_them(precision):
    """FP32: never, as they fit in the staging memory; FP64: not in an
    ensemble, and not once the launch shapes leave them unused"""
    plane = PLANE * (2 if precision == "fp64" else 1)
    with run(64, precision=precision) as r:  # (the library's code on the device before anything is measured)
        r.step(3)
    start = free()
    with run(0, precision=precision):
        plain = start - free()
    start = free()
    with run(64, precision=precision) as a, run(64, precision=precision) as b:
        if precision == "fp32":
            assert start - free() < 2 * plain + plane  # created
        with lb.Ensemble([a, b]) as e:
            e.step(24)
            e.sync()
        assert start - free() < 2 * plain + plane + (64 << 20)  # members (and the ensemble's own lists)
    start = free()
    with run(64, 9, precision) as r:  # two-step strips: particles in launches of their own
        r.step(30)
        r.sync()
        assert start - free() < plain + plane


def test_spare_slots_give_way():
    """post-stream populations with too little memory free beside the spare
    slots: given, and the run goes on as one that never had them"""
    import torch

    with run(64, 7, "fp64") as a, run(64, 7, "fp64") as b:
        a.set_pairs(0)
        for r in (a, b):
            r.step(21)
            r.sync()
        start = free()
        need = (2 * 9 * 8 + 2 * 9 * 8) * NX * NY
        hold = torch.empty(start - need + 2 * PLANE, dtype=torch.uint8, device="cuda")
        f, g = b.get_poststream()
        del hold
        torch.cuda.empty_cache()
        fa, ga = a.get_poststream()
        np.testing.assert_array_equal(f, fa)
        np.testing.assert_array_equal(g, ga)
        for n in (20, 3):
            a.step(n)
            b.step(n)
            for p, q in zip(a.get_populations(), b.get_populations()):
                np.testing.assert_array_equal(p, q)
            pa, pb = a.get_particles(), b.get_particles()
            for k in pa:
                np.testing.assert_array_equal(pb[k], pa[k], err_msg=k)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_transfers_beside_queued_steps(precision):
    """new populations and moments set while steps with riding particles are
    still queued: the steps before them, and what follows, as with a wait"""
    nx, ny, n = 1024, 512, 2000
    out = []
    for wait in (0, 1):
        with lb.Run(**lb.closure(nx, ny, Ra=1e6, Pr=1.0, U=0.1), precision=precision, nprtcl=n) as r:
            r.set_pair_shape(7)
            r.init_conduction(3, 5e-2)
            rng = np.random.default_rng(3)
            z = np.zeros(n)
            r.set_particles(np.arange(n, dtype=np.int32), rng.uniform(0.5, nx, n), rng.uniform(1.0, ny, n), z, z,
                            np.zeros(n, np.int32), z)
            r.step(20)
            f, g = r.get_populations()
            m = r.get_moments()
            for _ in range(5):
                r.step(100)
                if wait:
                    r.sync()
                r.set_populations(f, g)
                r.set_moments(m["rho"], m["u"], m["v"], m["T"])
            r.step(20)
            out.append((*r.get_populations(), *r.get_particles().values()))
    for p, q in zip(*out):
        np.testing.assert_array_equal(p, q)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("calls", [(2, 4, 6, 8, 10, 12, 14), (3, 5, 7, 9, 11, 21), (40, 33)])
@pytest.mark.parametrize("every", [0, 1, 2, 3, 7])
def test_riding_particles_over_call_lengths(precision, calls, every):
    """where a riding run ends (any call length, records that break it, a full
    ring that ends a call early) against single steps"""
    nx, ny, n = 128, 64, 96
    runs = []
    for pairs in (0, 1):
        r = lb.Run(**lb.closure(nx, ny, Ra=1e5, Pr=1.0, U=0.1), precision=precision, nprtcl=n, noutconfig=every,
                   record_slots=25, beta=0.5 if precision == "fp64" else 0.0)
        r.set_graph(0)
        r.set_pairs(pairs)
        if pairs:
            r.set_pair_shape(7)
        r.init_conduction(7, 5e-2)
        rng = np.random.default_rng(7)
        z = np.zeros(n)
        kinds = (np.arange(n) % 2).astype(np.int32)
        r.set_particles(np.arange(n, dtype=np.int32), rng.uniform(0.5, nx, n), rng.uniform(1.0, ny, n), z, z, kinds,
                        np.where(kinds == 1, 0.05, 0.0))
        runs.append(r)
    for steps in calls:
        out = []
        for r in runs:
            full = False
            try:
                r.step(steps)
            except lb.LbrbError:
                full = True
            p = r.get_particles()
            out.append((full, r.istep, p, r.drain_records_array(), r.get_populations()))
        (fa, ia, pa, ra, sa), (fb, ib, pb, rb, sb) = out
        assert (fa, ia) == (fb, ib)
        for k in pa:
            np.testing.assert_array_equal(pb[k], pa[k], err_msg=f"{k} after a call of {steps} steps")
        for x, y in zip(ra + sa, rb + sb):
            np.testing.assert_array_equal(y, x)
        # the next call reads u, v of this one's last step
    for r in runs:
        r.close()

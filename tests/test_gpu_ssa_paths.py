"""A cell's trajectory does not depend on how its CRUs are spread over CTAs and warps.

FP32 engine.

A CTA takes its CRUs on four lanes each (few of them), or in quiet passes followed by the CRUs that may
have a jump, each warp its own or queued for the event warps (the split between both following the
events); the flux sums are exact.  So every launch shape gives the same bits.

FP64 engine.  A CTA takes its CRUs on four lanes each or one, with the CRUs that have an event queued for
four lanes each (or, the queue full, at once).  The order of the flux sums follows the shape, but the CRUs
after one step depend on none: every shape gives their same bits.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def states(n, busy):
    from gwgb300 import engine

    rng = np.random.default_rng(n)
    ryr = np.zeros((n, 4, 6), np.int32)
    for j in range(4):
        k = rng.choice(6, (n, 5), p=[0.42, 0.02, 0.02, 0.1, 0.26, 0.18] if busy else [0.609, 0, 0, 0, 0.1955, 0.1955])
        for q in range(6):
            ryr[:, j, q] = (k == q).sum(1)
    lcc = rng.choice([1, 2, 3, 4, 5, 6, 9, 10, 11] if busy else [1, 2, 7], (n, 4)).astype(np.int32)
    cass = np.exp(rng.uniform(np.log(9e-5), np.log(6e-2), (n, 4))) if busy else np.full((n, 4), 1.4537e-4)
    return engine.CRUState(CaSS=cass.astype(np.float32).astype(float), LCC=lcc, RyR=ryr,
                           CaJSR=rng.uniform(0.6, 0.9, n).astype(np.float32).astype(float),
                           LCC_inactivation=(rng.random((n, 4)) < 0.85).astype(np.int32),
                           ClCh=(rng.random((n, 4)) < 0.05).astype(np.int32))


def simulate(n, busy, precision="fp32", steps=60, **shape):
    from gwgb300 import engine

    e = engine.Ensemble([n], precision=precision, seed=5, **shape)
    if busy:
        g = e.get_globals(0)
        g[0], g[3], g[4] = -3.7, 4.0e-4, 0.88
        e.set_globals(0, g)
    e.set_crus(0, states(n, busy))
    e.set_pulse(0.0, 500.0, 0.5, 100.0)
    e.run(1e-3, steps)
    s = e.get_crus(0)
    out = {k: np.array(getattr(s, k)) for k in ("CaSS", "CaJSR", "LCC", "LCC_inactivation", "RyR", "ClCh")}
    out["globals"] = e.get_globals(0)
    out["carry"] = np.array(e.get_flux_carry(0))
    out["events"] = np.array(e.stats()["events"])
    return out


@pytest.mark.parametrize("busy", [False, True])
@pytest.mark.parametrize("n,shapes", [
    (5, [(2, 0)]),                          # part of one group of eight
    (129, [(2, 0), (5, 0)]),                # one more than a pass of 16 warps
    (257, [(2, 0), (1, 320), (3, 0)]),      # one more than a CTA of 16 warps takes without a queue
    (385, [(1, 416), (2, 0), (4, 128)]),    # one more than a CTA of 12 warps does
    (1000, [(1, 1024), (2, 0), (4, 0), (9, 0), (16, 0)]),
    (2080, [(1, 2080), (2, 1056), (3, 0)]),  # many groups per warp, a full queue when busy
])
def test_every_shape_gives_the_same_bits(n, shapes, busy):
    want = simulate(n, busy, cluster_ctas=0)
    assert not busy or want["events"] > 2 * n
    for cl, tile in shapes:
        got = simulate(n, busy, cluster_ctas=cl, cta_crus=tile)
        for k in want:
            assert np.array_equal(want[k], got[k]), (k, cl, tile)


@pytest.mark.parametrize("busy", [False, True])
@pytest.mark.parametrize("n,shapes", [
    (7, [(2, 0)]),                          # part of one group of eight
    (65, [(1, 96), (2, 64)]),               # one more than a pass of eight warps
    (385, [(1, 416), (2, 0), (4, 0)]),      # one more than the CTAs of four lanes per CRU take
    (1100, [(1, 1120), (2, 576), (4, 288)]),  # more events than the queue holds when busy
])
def test_every_shape_gives_the_same_crus_fp64(n, shapes, busy):
    want = simulate(n, busy, precision="fp64", steps=1, cluster_ctas=0)
    for cl, tile in shapes:
        got = simulate(n, busy, precision="fp64", steps=1, cluster_ctas=cl, cta_crus=tile)
        for k in ("CaSS", "CaJSR", "LCC", "LCC_inactivation", "RyR", "ClCh", "events"):
            assert np.array_equal(want[k], got[k]), (k, cl, tile)


def test_many_events_in_one_warp():
    """A step in which an event warp takes more than 500 CRUs of a CTA (large steps, and more than a third of the
    CRUs with a jump when the split still expects one in 32): the same bits in every shape, and again."""
    from gwgb300 import engine

    n, dt = 2080, 1.5e-2

    def run(steps, **shape):
        with engine.Ensemble([n], precision="fp32", seed=6, **shape) as e:
            g = e.get_globals(0)
            g[0], g[3], g[4] = 20.0, 4.0e-4, 0.88
            e.set_globals(0, g)
            e.set_crus(0, states(n, True))
            e.run(dt, steps)
            s = e.get_crus(0)
            return ([np.array(getattr(s, k)) for k in ("CaSS", "CaJSR", "LCC", "RyR", "ClCh")] +
                    [e.get_globals(0), np.array(e.get_flux_carry(0))]), e.stats()["events"]

    assert run(1)[1] > 1200
    want, _ = run(12)
    for shape in (dict(cluster_ctas=1, cta_crus=2080), dict(cluster_ctas=1, cta_crus=2080), dict(cluster_ctas=2), dict(cluster_ctas=3)):
        got, _ = run(12, **shape)
        for a, b in zip(want, got):
            assert np.array_equal(a, b), shape

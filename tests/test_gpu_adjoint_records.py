"""The reverse sweep of CRUs with jumps, from sub-steps recorded ahead of it or re-run in it.

ClCh gates that flip about twelve times per CRU-step: a segment of twelve steps has more sub-steps than
the pool of records holds, a segment of one fits, and some steps have more than one record block in both.
All are the same arithmetic, so the sensitivities are the same bits.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flips", [1.0, 4000.0])
def test_recorded_and_rerun_steps_agree(flips):
    from gwgb300 import engine
    from gwgb300.adjoint import GradEngine

    ncru, steps = [60, 37], 12
    p = engine.params_from(None, kfClCh=flips / 1.5e-4, kbClCh=flips)
    got = {}
    for every in (12, 1):
        with GradEngine(ncru, p, n_steps=steps, dt=1.5e-3, seed=3, sample_every=1, checkpoint_every=every) as e:
            for c, n in enumerate(ncru):
                r = np.random.default_rng(c)
                ryr = np.zeros((n, 4, 6), np.int32)
                k = r.choice(6, (n, 4, 5), p=[0.5, 0, 0, 0.1, 0.2, 0.2])
                for q in range(6):
                    ryr[:, :, q] = (k == q).sum(2)
                s = engine.CRUState(CaSS=np.full((n, 4), 1.5e-4), CaJSR=np.full(n, 0.9), RyR=ryr,
                                    LCC=r.choice([1, 2, 3, 5, 6], (n, 4)).astype(np.int32),
                                    LCC_inactivation=(r.random((n, 4)) < 0.9).astype(np.int32),
                                    ClCh=(r.random((n, 4)) < 0.5).astype(np.int32))
                with engine.Ensemble([n], precision="fp64") as ens:
                    g = ens.get_globals(0)
                e.set_state(c, g, s)
            V = e.forward()
            got[every] = V, e.backward(np.random.default_rng(1).normal(size=V.shape)), e.stats()["events"]
    assert got[12][2] == got[1][2] and (flips < 2 or got[12][2] > 8 * steps * sum(ncru))
    assert np.array_equal(got[12][0], got[1][0])
    assert np.all(np.isfinite(got[12][1])) and np.any(got[12][1] != 0)
    assert np.array_equal(got[12][1], got[1][1])

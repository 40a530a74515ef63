"""A launch whose per-step data stop coming ends by itself on every SSA path: the test hook makes the leader's wait
for the partials of step 0 expect bytes that no one sends; the leader stops, the SSA values of step 2 never come, and
all warps of every CTA of the cell stop together (in a split CTA the event warps by the quiet ones' decision)."""
import time

import numpy as np
import pytest
from test_gpu_ssa_paths import states

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,precision,shape", [
    (60, "fp32", dict(cluster_ctas=1)),                   # four lanes per CRU
    (200, "fp32", dict(cluster_ctas=1, cta_crus=224)),    # a lane per CRU
    (700, "fp32", dict(cluster_ctas=1)),                  # split, one CTA
    (1100, "fp32", dict(cluster_ctas=2)),                 # split, two CTAs
    (100, "fp64", dict(cluster_ctas=2)),
])
def test_stops_within_seconds(monkeypatch, n, precision, shape):
    from gwgb300 import Ensemble, _lib

    monkeypatch.setenv("GWGB300_TEST_SYNC_TIMEOUT", "2")
    with Ensemble([n], precision=precision, seed=1, **shape) as e:
        e.set_crus(0, states(n, True))
        t = time.monotonic()
        with pytest.raises(_lib.GWError) as ex:
            e.run(1e-3, 30)
        assert ex.value.code == _lib.GW_ERR_SYNC_TIMEOUT and time.monotonic() - t < 30
    monkeypatch.delenv("GWGB300_TEST_SYNC_TIMEOUT")
    with Ensemble([n], precision=precision, seed=1, **shape) as e:
        e.set_crus(0, states(n, True))
        e.run(1e-3, 30)
        assert np.all(np.isfinite(e.get_globals(0)))

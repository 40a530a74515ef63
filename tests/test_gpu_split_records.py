"""Records and repeatability of the FP32 path of CTAs with many CRUs, whose warps are split between quiet passes and
events: cells of 500 to 1,600 CRUs held by one or two CTAs, amid the release, recorded every few steps while the split
follows the events, against the same run spread over CTAs of few CRUs (another path, same bits)."""
import numpy as np
import pytest
from test_gpu_records import _ryr_code, _sums_from_arrays
from test_gpu_ssa_paths import states

pytestmark = pytest.mark.gpu


def _run(n, every, steps, cluster_ctas, dt=1e-3, codec=False):
    from gwgb300 import engine

    with engine.Ensemble([n], precision="fp32", seed=8, cluster_ctas=cluster_ctas) as e:
        g = e.get_globals(0)
        g[0], g[3], g[4] = -85.0, 1.6e-4, 0.88
        e.set_globals(0, g)
        # closed channels (about one CRU in a hundred has a jump in a step) and, every 200 steps, V up to 150 mV and
        # back after 60 (LCC activation: about one in eight), so that the split follows a load that rises and falls
        init = states(n, False)
        init.LCC[:], init.RyR[:], init.RyR[:, :, 0], init.ClCh[:] = 1, 0, 5, 0
        e.set_crus(0, init)
        k = np.arange(steps) % 200
        e.set_samples(np.where((k >= 60) & (k < 70), 23500.0, 0.0) - np.where((k >= 120) & (k < 130), 23500.0, 0.0))
        tr = e.run(dt, steps, record_every=every, cru_cell=0, sums=True, codec=codec)
        s = e.get_crus(0)
        end = {k: np.array(getattr(s, k)) for k in ("CaSS", "CaJSR", "LCC", "LCC_inactivation", "RyR", "ClCh")}
        end["globals"], end["carry"] = e.get_globals(0), np.array(e.get_flux_carry(0))
        return tr, end


@pytest.mark.parametrize("n,every,ctas", [(500, 1, 1), (1100, 1, 1), (1600, 3, 1), (1100, 1, 2)])  # of 12, or 12 and 16 warps
def test_records_equal_those_of_few_crus_per_cta(n, every, ctas):
    steps = 480
    a, end_a = _run(n, every, steps, 16)
    b, end_b = _run(n, every, steps, ctas)
    c, _ = _run(n, every, steps, ctas, codec=True)
    for k in end_a:
        np.testing.assert_array_equal(end_a[k], end_b[k], err_msg=k)
    np.testing.assert_array_equal(a.globals, b.globals)
    for k in a.crus:
        np.testing.assert_array_equal(a.crus[k], b.crus[k], err_msg=k)
    np.testing.assert_array_equal(a.cru_sums, b.cru_sums)
    np.testing.assert_array_equal(b.cru_sums, c.cru_sums)
    want = _sums_from_arrays(b.crus)
    for f in (0, 1, 3, 4, 7):
        np.testing.assert_array_equal(b.cru_sums[0][:, f], want[:, f])
    np.testing.assert_array_equal(c.codec["RyR"], _ryr_code(b.crus["RyR"]))
    np.testing.assert_array_equal(c.codec["LCC"], b.crus["LCC"].astype(np.int8))
    np.testing.assert_array_equal(c.codec["CaSS"], b.crus["CaSS"].astype(np.float32))
    np.testing.assert_array_equal(c.codec["CaJSR"], b.crus["CaJSR"].astype(np.float32))
    # the load the split follows: CRUs whose LCCs change between records
    d = (np.diff(b.crus["LCC"], axis=0) != 0).any(axis=2).sum(axis=1)
    assert d.max() > 4 * np.median(d[:20]), (d.max(), np.median(d[:20]))


def test_runs_repeat():
    a, end_a = _run(1600, 7, 480, 1)
    b, end_b = _run(1600, 7, 480, 1)
    for k in end_a:
        np.testing.assert_array_equal(end_a[k], end_b[k], err_msg=k)
    np.testing.assert_array_equal(a.cru_sums, b.cru_sums)
    np.testing.assert_array_equal(a.globals, b.globals)

"""Ensembles of so many small FP32 cells that several CTAs share an SM and a CTA has one or two SSA warps:
every cell as it runs alone (its CTAs then have more warps), bit for bit."""
import numpy as np
import pytest
from test_gpu_ssa_paths import states

pytestmark = pytest.mark.gpu

CELLS = 160


def _fill(e, i, n, busy):
    s = states(n, busy)
    s.ClCh = (np.random.default_rng(n).random((n, 4)) < 0.4).astype(np.int32)
    if busy:
        g = e.get_globals(i)
        g[0], g[3], g[4] = -3.7, 4.0e-4, 0.88
        e.set_globals(i, g)
    e.set_crus(i, s)


def _state(e, i):
    s = e.get_crus(i)
    out = {k: np.array(getattr(s, k)) for k in ("CaSS", "CaJSR", "LCC", "LCC_inactivation", "RyR", "ClCh")}
    out["globals"], out["carry"] = e.get_globals(i), np.array(e.get_flux_carry(i))
    return out


@pytest.mark.parametrize("busy", [False, True])
@pytest.mark.parametrize("largest", [32, 60, 100])
def test_each_cell_as_alone(largest, busy):
    from gwgb300 import engine

    ncru = [5 + (7 * i) % (largest - 4) for i in range(CELLS - 1)] + [largest]
    with engine.Ensemble(ncru, precision="fp32", seed=5) as e:
        for i, n in enumerate(ncru):
            _fill(e, i, n, busy)
        e.set_pulse(0.0, 500.0, 0.5, 100.0)
        e.run(1e-3, 40)
        assert e.stats()["ctas"] > 152 and (not busy or e.stats()["events"] > sum(ncru))
        got = {i: _state(e, i) for i in list(range(0, CELLS, 9)) + [CELLS - 1]}
    for i, g in got.items():
        with engine.Ensemble([ncru[i]], precision="fp32", seed=5, cell_base=i) as e:
            _fill(e, 0, ncru[i], busy)
            e.set_pulse(0.0, 500.0, 0.5, 100.0)
            e.run(1e-3, 40)
            want = _state(e, 0)
        for k in want:
            assert np.array_equal(want[k], g[k]), (i, ncru[i], k)

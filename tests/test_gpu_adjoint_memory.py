"""The optional records of the gradient's reverse sweep take at most a quarter of the device memory that the rest
leaves: with the card nearly full they shrink, and the sensitivities stay the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, S, STEPS = 30000, 400, 10  # CRUs, steps of a segment, steps of the run


def _engine():
    from gwgb300.adjoint import GradEngine

    return GradEngine([N], None, n_steps=STEPS, seed=2, sample_every=1, checkpoint_every=S)


def _sens(e):
    from gwgb300 import _lib, engine

    r = np.random.default_rng(0)
    ryr = np.zeros((N, 4, 6), np.int32)
    k = r.choice(6, (N, 4, 5), p=[0.42, 0.02, 0.02, 0.1, 0.26, 0.18])
    for q in range(6):
        ryr[:, :, q] = (k == q).sum(2)
    e.set_state(0, _lib.default_globals(py=True), engine.CRUState(
        CaSS=np.exp(r.uniform(np.log(9e-5), np.log(6e-2), (N, 4))), CaJSR=r.uniform(0.6, 0.9, N), RyR=ryr,
        LCC=r.choice([1, 2, 3, 5, 6], (N, 4)).astype(np.int32),
        LCC_inactivation=(r.random((N, 4)) < 0.9).astype(np.int32), ClCh=np.zeros((N, 4), np.int32)))
    V = e.forward()
    return V, e.backward(np.random.default_rng(1).normal(size=V.shape))


def test_records_leave_memory():
    import torch

    gb = 1 << 30
    with _engine() as e:
        full = e.stats()["segment_bytes"]
        want = _sens(e)
    pool = N * S // 4 * 128  # records of 128 bytes for a quarter of the CRU-steps
    fill = None
    got = {}
    for left in (full - pool + 0.9 * gb, full - pool + 0.12 * gb):  # the required arrays, and something
        fill = None
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        fill = torch.empty(int(free - left), dtype=torch.uint8, device="cuda")
        with _engine() as e:
            rest, seg = torch.cuda.mem_get_info()[0], e.stats()["segment_bytes"]
            got[left] = seg
            taken = seg - (full - pool - 4 * N * S - 4)  # by the records, their index and their count
            assert 0 <= taken <= 0.26 * (rest + taken) + (8 << 20)
            V, sens = _sens(e)
        assert np.array_equal(V, want[0]) and np.array_equal(sens, want[1])
    del fill
    torch.cuda.empty_cache()
    assert full > max(got.values()) and min(got.values()) < max(got.values())

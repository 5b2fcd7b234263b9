"""The two-steps-a-pass kernel (lbm_pair.cuh) on domains on which lbm_run would
not use it, through lbm_selftest_pair_steps: boxes a cell thick, one cell either
side of whole tiles of 64 x 8 and 64 x 10 and of whole z chunks, all storages,
from a step counter that is not zero; and the bounded waits of its copies, made
to run out at any place of a block's work."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

OK, UNSUPPORTED, TIMEOUT = 0, 5, 11


def _solver(n, storage, lid="injection"):
    from cavityflow_cuda_gb300 import CLbmSolverGB300

    _, itau = orc.tau_of(0.0192, np.float32)
    return CLbmSolverGB300(n, itau, np.float32(0.08), storage=storage, lid=lid)


def _state(n, seed):
    rng = np.random.default_rng(seed)
    w = np.array([1 / 18] * 4 + [1 / 36] * 12 + [1 / 18] * 2 + [1 / 3], dtype=np.float32)
    noise = rng.random((19, n[2] + 2, n[1] + 2, n[0] + 2), dtype=np.float32)
    return w[:, None, None, None] * (np.float32(0.98) + np.float32(0.04) * noise)


SHAPES = [((1, 1, 1), "injection"), ((1, 30, 40), "wall"), ((40, 1, 33), "injection"), ((70, 23, 1), "wall"),
          ((63, 9, 31), "injection"), ((64, 10, 32), "wall"), ((65, 11, 33), "injection"), ((64, 8, 65), "injection"),
          ((129, 17, 9), "wall"), ((200, 21, 64), "injection")]


@pytest.mark.parametrize("storage", ["f32", "f16s", "bf16s", "f16sr"])
@pytest.mark.parametrize("n,lid", SHAPES)
def test_forced_pairs_match_single_steps(gpu, storage, n, lid):
    from cavityflow_cuda_gb300 import kernel_launches

    start, got = _state(n, 11), []
    for forced in (True, False):
        with _solver(n, storage, lid) as s:
            s.set_all(start)
            for i in range(2 + 4 + 2 + 8 + 1):
                if forced and i in (2, 8):
                    before = kernel_launches()
                    assert s._lib.lbm_selftest_pair_steps(s._h, 1 if i == 2 else 2, -1) == OK
                    assert kernel_launches() - before == (2 if i == 2 else 4)
                elif not forced or i in (0, 1, 6, 7, 16):
                    (s.simulationStepBeta if i & 1 else s.simulationStepAlpha)()
            assert s.info()["step_counter"] == 17
            if forced:
                assert s._lib.lbm_selftest_pair_steps(s._h, 1, -1) == UNSUPPORTED  # the next step is beta
            got.append(s.get_all())
    assert np.array_equal(got[0].view(np.uint32), got[1].view(np.uint32))


@pytest.mark.parametrize("storage", ["f32", "f16sr"])
def test_expired_wait_is_reported_and_the_solver_stays_usable(gpu, storage):
    """Limits below and around the time of a copy: blocks give up on their first fill, on later ones, or not
    at all.  Every launch ends, the failure is reported once, and the counters that blocks share are as the next
    launch wants them."""
    n = (200, 160, 96)
    start = _state(n, 5)
    with _solver(n, storage) as s:
        s.set_all(start)
        assert s._lib.lbm_selftest_pair_steps(s._h, 2, -1) == OK
        want = s.get_all()
        seen = set()
        for limit in (0, 400, 800, 1200, 1600, 2000, 2500, 3000, 4000):
            status = s._lib.lbm_selftest_pair_steps(s._h, 1, limit)
            assert status in (OK, TIMEOUT), s._lib.lbm_last_error()
            assert limit > 0 or status == TIMEOUT
            seen.add(status)
            assert s._lib.lbm_synchronize(s._h) == OK
        assert TIMEOUT in seen
    with _solver(n, storage) as s:  # a launch after one that gave up
        assert s._lib.lbm_selftest_pair_steps(s._h, 1, 0) == TIMEOUT
        s.run((-s.info()["step_counter"]) % 4)
        s.set_all(start)
        with _solver(n, storage) as t:
            t.set_all(start)
            assert t._lib.lbm_selftest_pair_steps(t._h, 2, -1) == OK
            fresh = t.get_all()
        assert np.array_equal(fresh.view(np.uint32), want.view(np.uint32))
        if storage == "f32":  # the stochastic storage's dither depends on the step
            assert s._lib.lbm_selftest_pair_steps(s._h, 2, -1) == OK
            assert np.array_equal(s.get_all().view(np.uint32), want.view(np.uint32))

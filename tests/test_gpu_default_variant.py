"""The 16-bit storages' default launch variant follows the domain's size; at
both sides of each border the steps (replayed graph and single launches) equal
the oracle bit for bit."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

SIZES = [((56, 55, 55), 6), ((56, 56, 55), 8), ((103, 103, 103), 8), ((104, 103, 103), 23), ((124, 124, 123), 23),
         ((124, 124, 124), 20)]


@pytest.mark.parametrize("storage,kind", [("f16s", 0), ("bf16s", 1), ("f16sr", 2)])
@pytest.mark.parametrize("n,variant", SIZES)
def test_default_variant_matches_oracle(gpu, oracle, storage, kind, n, variant):
    from cavityflow_cuda_gb300 import CLbmSolverGB300

    _, itau = orc.tau_of(0.0192, np.float32)
    lid = np.float32(0.08)
    small = n[0] < 60
    steps = 64 + 3 if small else 3  # 64: a replayed graph
    dd, _ = oracle.run_cavity_s(*n, kind, itau, lid, steps)
    want = oracle.unshift(dd, kind)
    with CLbmSolverGB300(n, itau, lid, storage=storage) as s:
        assert s.info()["fast_variant"] == variant
        s.run(steps - 3)
        s.simulationStepAlpha()
        s.simulationStepBeta()
        s.run(1)
        assert np.array_equal(s.get_all().view(np.uint32), want.view(np.uint32))

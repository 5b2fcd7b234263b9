"""The FP64 collision on the integer units (lbm_f64.cuh) where operands leave the
range of its integer products: cells at rest, planes of symmetry, tiny, huge,
zero and non-finite populations, next to ordinary ones.  Bit-identical to the
oracle (any NaN equals any NaN)."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

W = np.array([1 / 18] * 4 + [1 / 36] * 12 + [1 / 18] * 2 + [1 / 3])
SPECIAL = [0.0, -0.0, 5e-324, 1e-310, 1e-300, 1e-160, -1e-120, 1e120, -1e160, 1e300, np.inf, -np.inf, np.nan]


@pytest.mark.parametrize("variant", [-1, 1, 8, 25])
@pytest.mark.parametrize("kind", ["special", "scaled", "symmetric"])
def test_out_of_range_operands_match_oracle(gpu, oracle, variant, kind):
    from cavityflow_cuda_gb300 import CLbmSolverGB300

    n = (21, 10, 9)
    _, itau = orc.tau_of(0.0192, np.float64)
    rng = np.random.default_rng(5)
    dd = W[:, None, None, None] * (0.98 + 0.04 * rng.random((19, n[2] + 2, n[1] + 2, n[0] + 2)))
    if kind == "special":  # one population in forty of an odd kind
        pick = rng.random(dd.shape) < 1 / 40
        dd[pick] = np.array(SPECIAL)[rng.integers(0, len(SPECIAL), int(pick.sum()))]
    elif kind == "scaled":  # whole cells at other magnitudes, over the ends of the accepted exponents
        dd *= 2.0 ** rng.integers(-1000, 600, dd.shape[1:])
    else:  # populations equal in pairs along x and z: those velocity components are exactly zero
        for k in (0, 8, 10, 12, 14, 16, 4, 6):
            dd[k + 1] = dd[k]
    with CLbmSolverGB300(n, itau, 0.05, storage="f64", fast_variant=variant) as s:
        s.set_all(dd)
        flags = s.flags_all()
        s.run(3)
        got = s.get_all()
    want = dd.copy()
    for i in range(3):
        oracle.step(want, flags, i, itau, 0.05)
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got[~nan].view(np.uint64), want[~nan].view(np.uint64))

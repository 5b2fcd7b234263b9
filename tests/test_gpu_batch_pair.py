"""LbmBatch.run's two-steps-a-pass kernel (lbm_pair.cuh), bit-identical to the
batch's single-step kernels, which the other tests hold to single solvers and
those to the oracle: rows of one tile and of several, partial tiles and z chunks,
boxes a cell thick, runs from either step parity, every cell and wall slot
disturbed."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

ODD = [(1, 1, 1), (1, 40, 9), (2, 3, 70), (7, 65, 33), (33, 1, 64), (63, 8, 32), (64, 9, 1), (65, 17, 65), (96, 41, 34),
       (97, 11, 66), (129, 30, 31), (16, 16, 16), (18, 96, 20)]


def _state(n, seed):
    rng = np.random.default_rng(seed)
    w = np.array([1 / 18] * 4 + [1 / 36] * 12 + [1 / 18] * 2 + [1 / 3], dtype=np.float32)
    noise = rng.random((19, n[2] + 2, n[1] + 2, n[0] + 2), dtype=np.float32)
    return w[:, None, None, None] * (np.float32(0.98) + np.float32(0.04) * noise)


@pytest.mark.parametrize("rest,count", [((64, 64, 64), 24), ((48, 40, 37), 90)])
def test_batch_pairs_match_single_steps(gpu, rest, count):
    from cavityflow_cuda_gb300 import kernel_launches
    from cavityflow_cuda_gb300.solver import LbmBatch

    sizes = ODD[:7] + [rest] * count + ODD[7:]
    _, itau = orc.tau_of(0.0192, np.float32)
    doms = [(n, float(itau) * (1 - 0.001 * (i % 7)), 0.02 + 0.005 * (i % 11)) for i, n in enumerate(sizes)]
    checked = [i for i, n in enumerate(sizes) if n != rest or i in (7, 6 + count)]
    runs = (5, 1, 10, 2)  # from an even and an odd counter, with and without a rest
    got = []
    for separate in (False, True):
        with LbmBatch(doms, storage="f32") as b:
            if separate:
                b.set_fast_variant(b.info()["fast_variant"])
            for i in checked:
                b.domain(i).set_all(_state(sizes[i], i))
            before = kernel_launches()
            for r in runs:
                b.run(r)
            launched = kernel_launches() - before
            assert (launched == sum(runs)) if separate else (launched == sum(runs) - 6)
            got.append([b.domain(i).get_all() for i in checked])
    for i, a, c in zip(checked, *got):
        assert np.array_equal(a.view(np.uint32), c.view(np.uint32)), sizes[i]

"""lbm_run's two-steps-a-pass kernel (lbm_pair.cuh), bit-identical to the oracle
(FP32) and to the single-step kernels, which the other tests hold to the oracle
(16-bit storages): domains with partial tiles on every axis, both lids, runs
from either step parity, starting from a disturbed state in every cell and
wall slot."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _solver(n, storage, itau, lid_u, lid="injection", **kw):
    from cavityflow_cuda_gb300 import CLbmSolverGB300

    return CLbmSolverGB300(n, itau, lid_u, storage=storage, lid=lid, **kw)


def same_bits(a, b):
    return a.shape == b.shape and np.array_equal(np.ascontiguousarray(a).view(np.uint8),
                                                  np.ascontiguousarray(b).view(np.uint8))


def _state(n, seed):
    """Populations near rest, every cell and halo slot disturbed (reference layout)."""
    rng = np.random.default_rng(seed)
    w = np.array([1 / 18] * 4 + [1 / 36] * 12 + [1 / 18] * 2 + [1 / 3], dtype=np.float32)
    noise = rng.random((19, n[2] + 2, n[1] + 2, n[0] + 2), dtype=np.float32)
    return w[:, None, None, None] * (np.float32(0.98) + np.float32(0.04) * noise)


# One cell beyond whole tiles of 64 x 8 (64 x 10) and beyond whole z chunks (129 is too narrow for the pair kernel to pay, 449
# is not); whole tiles; one tile less a cell; larger, where it pays for the storages that round to nearest; larger
# still for the stochastic one.
SHAPES = [((129, 121, 131), "injection"), ((449, 121, 131), "injection"), ((192, 128, 97), "wall"),
          ((383, 63, 90), "injection"), ((320, 257, 249), "injection")]


@pytest.mark.parametrize("storage,n,lid", [(st, *shape) for shape in SHAPES for st in ("f32", "f16s", "bf16s")] +
                         [("f16sr", (448, 383, 201), "wall")])
def test_pairs_match_single_steps(gpu, oracle, storage, n, lid):
    from cavityflow_cuda_gb300 import kernel_launches

    _, itau = orc.tau_of(0.0192, np.float32)
    lid_u = np.float32(0.08)
    big = n[0] * n[1] * n[2] > 10_000_000
    runs = (5,) if big else (1, 6, 10)  # from an even and from an odd counter, with and without a rest
    start = _state(n, 7)
    with _solver(n, storage, itau, lid_u, lid) as s:
        s.set_all(start)
        saved = 0
        for r in runs:
            before = kernel_launches()
            s.run(r)
            saved += r - (kernel_launches() - before)
        got = s.get_all()
        flags = s.flags_all()
    if big or (storage == "f32" and n[0] != 129):
        assert saved > 0, "the domain should be large enough for two steps a pass"
    if storage == "f32":
        want = start.copy()
        for i in range(sum(runs)):
            oracle.step(want, flags, i, itau, lid_u, wall=lid == "wall")
    else:
        with _solver(n, storage, itau, lid_u, lid) as s:
            s.set_all(start)
            for i in range(sum(runs)):
                (s.simulationStepBeta if i & 1 else s.simulationStepAlpha)()
            want = s.get_all()
    assert same_bits(got, want), (storage, n)


def test_chosen_variant_and_capture_keep_single_steps(gpu):
    """A solver with a launch variant of its own takes one step a launch, and so
    does a run captured into the caller's graph; both give the same state."""
    import torch

    from cavityflow_cuda_gb300 import kernel_launches

    n = (130, 127, 128)
    _, itau = orc.tau_of(0.0192, np.float32)
    with _solver(n, "f32", itau, 0.05) as a, _solver(n, "f32", itau, 0.05, fast_variant=13) as b, \
            _solver(n, "f32", itau, 0.05) as c:
        before = kernel_launches()
        a.run(8)
        assert kernel_launches() - before == 4
        before = kernel_launches()
        b.run(8)
        assert kernel_launches() - before == 8
        st = torch.cuda.Stream()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            c.run(8, stream=st)
        g.replay()
        torch.cuda.synchronize()
        want = b.get_all()
        assert same_bits(a.get_all(), want) and same_bits(c.get_all(), want)
        a.set_fast_variant(13)
        before = kernel_launches()
        a.run(8)
        assert kernel_launches() - before == 8
        b.run(8)
        assert same_bits(a.get_all(), b.get_all())


@pytest.mark.parametrize("storage", ["f32", "f16s", "bf16s", "f16sr"])
def test_pairs_with_odd_rows(gpu, storage):
    """Rows of an odd number of cells, whose last pair of cells is one cell and
    the wall, and the wall slots of all six faces."""
    from cavityflow_cuda_gb300 import kernel_launches

    n = (447, 300, 200)
    _, itau = orc.tau_of(0.0192, np.float32)
    start = _state(n, 3)
    got = []
    for launches, variant in ((3, {}), (5, {"fast_variant": 13})):  # two steps a pass, single steps
        with _solver(n, storage, itau, 0.08, "wall", **variant) as s:
            s.set_all(start)
            before = kernel_launches()
            s.run(5)
            assert kernel_launches() - before == launches
            got.append(s.get_all())
    assert same_bits(*got)

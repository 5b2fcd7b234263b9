"""The host side of the two-steps-a-pass runs and of the packed getters, on a GPU:
captures on this and on other streams, streams and threads that share a packing
buffer."""
import threading

import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

BIG, SMALL = (130, 127, 128), (37, 25, 41)


def _solver(n, storage="f32"):
    from cavityflow_cuda_gb300 import CLbmSolverGB300

    _, itau = orc.tau_of(0.0192, np.float32)
    return CLbmSolverGB300(n, itau, np.float32(0.05), storage=storage)


def _batch():
    from cavityflow_cuda_gb300 import LbmBatch

    return LbmBatch([((64, 64, 64), 1.6 + 0.001 * i, 0.05) for i in range(40)], storage="f32")


def same(a, b):
    return np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("kind", ["solver", "batch"])
def test_run_beside_a_capture_on_another_stream(gpu, kind):
    """The first run that takes two steps a pass allocates; a capture in global mode on another stream survives it."""
    import torch

    from cavityflow_cuda_gb300 import kernel_launches

    a, b = (_solver(BIG), _solver(BIG)) if kind == "solver" else (_batch(), _batch())
    x = torch.ones(8, device="cuda")
    st, other = torch.cuda.Stream(), torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    before = kernel_launches()
    with torch.cuda.graph(g, stream=st, capture_error_mode="global"):
        x += 1
        a.run(8, stream=other)
    assert kernel_launches() - before == 4
    g.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [2.0] * 8
    b.set_fast_variant(b.info()["fast_variant"])
    b.run(8)
    va, vb = (a, b) if kind == "solver" else (a.domain(17), b.domain(17))
    assert same(va.get_all(), vb.get_all())
    a.close()
    b.close()


def test_captured_batch_run_replays_single_steps(gpu):
    import torch

    with _batch() as a, _batch() as b:
        b.set_fast_variant(b.info()["fast_variant"])
        st = torch.cuda.Stream()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            a.run(6, stream=st)
        g.replay()
        torch.cuda.synchronize()
        b.run(6)
        for i in (0, 39):
            assert same(a.domain(i).get_all(), b.domain(i).get_all())


@pytest.mark.parametrize("storage", ["f32", "f16sr"])
def test_populations_getter_on_a_capturing_stream(gpu, storage):
    """No packing buffer in the caller's graph: row-wise copies (FP32) or the staging buffer (16 bits), which the
    solver holds from a call before."""
    import torch

    with _solver(SMALL, storage) as s:
        s.run(7)
        want = s.get_all()
        sub = np.ascontiguousarray(want[:, 2:7, 3:9, 1:13])
        out = torch.zeros(sub.shape, dtype=torch.float32, pin_memory=True)
        box = (1, 3, 2), (12, 6, 5)
        if storage != "f32":
            s.set_all(want)  # makes the staging buffer
        st = torch.cuda.Stream()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            s.getDensityDistributions(*box, out=out.numpy(), stream=st, sync=False)
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert same(out.numpy(), sub)


def test_streams_and_threads_share_a_packing_buffer(gpu):
    """Asynchronous getters of one solver on several streams, and of a batch's domains on several threads, all take
    the same buffer: none may see another's values."""
    import torch

    with _solver(SMALL) as s:
        s.run(11)
        want = s.get_all()
        streams = [torch.cuda.Stream() for _ in range(4)]
        boxes = [((1, 1, 1 + 3 * i), (37, 25, 3 + i)) for i in range(8)]
        outs = [torch.zeros((19, n[2], n[1], n[0]), dtype=torch.float32, pin_memory=True) for _, n in boxes]
        torch.cuda.synchronize()
        for _ in range(5):
            for i, (box, o) in enumerate(zip(boxes, outs)):
                s.getDensityDistributions(*box, out=o.numpy(), stream=streams[i % 4], sync=False)
        torch.cuda.synchronize()
        for (o, n), got in zip(boxes, outs):
            assert same(got.numpy(), np.ascontiguousarray(
                want[:, o[2]:o[2] + n[2], o[1]:o[1] + n[1], o[0]:o[0] + n[0]])), o
    with _batch() as b:
        b.run(9)
        views = [b.domain(i) for i in range(8)]
        want = [(v.getDensities(), v.getVelocities(), v.getDensityDistributions()) for v in views]
        bad = []

        def work(i):
            for _ in range(10):
                got = views[i].getDensities(), views[i].getVelocities(), views[i].getDensityDistributions()
                if not all(same(x, y) for x, y in zip(got, want[i])):
                    bad.append(i)

        threads = [threading.Thread(target=work, args=(i,)) for i in range(8)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not bad

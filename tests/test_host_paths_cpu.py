"""The host code around the two-steps-a-pass kernels and the getters, on a
stand-in for the CUDA runtime (tests/fake/cudart.c) in a process of its own:
memory that runs out, launches and copies that fail, captures on other streams,
other threads.  Kernels do nothing there, so these tests say nothing about
results."""
import os
import shutil
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA_INCLUDE = "/usr/local/cuda/include"

PREAMBLE = """
import ctypes as C, threading, time
import numpy as np
from cavityflow_cuda_gb300 import CLbmSolverGB300, LbmBatch, LbmError, LbmServer, kernel_launches
from cavityflow_cuda_gb300.solver import load_library
lib = load_library()
fake = C.CDLL(None)
fake.fake_used.restype = C.c_size_t
fake.fake_memory.argtypes = [C.c_size_t]
fake.fake_live.argtypes = [C.c_void_p]
fake.fake_capturing.argtypes = [C.c_void_p]
MB, GB = 1 << 20, 1 << 30
TIMEOUT = 11
def solver(n=(256, 256, 256), storage="f32", **kw):
    return CLbmSolverGB300(n, 1.6, 0.05, storage=storage, **kw)
def batch(n=(64, 64, 64), count=76, storage="f32"):
    return LbmBatch([(n, 1.6, 0.05)] * count, storage=storage)
def run(s, steps):  # launches of a run
    before = kernel_launches()
    s.run(steps)
    return kernel_launches() - before
LaunchFn = C.CFUNCTYPE(None, C.c_char_p, C.POINTER(C.c_void_p))
def watch(f):  # f(kernel name, args) before each launch
    global _cb
    _cb = LaunchFn(f)
    fake.fake_on_launch(_cb)
"""


@pytest.fixture(scope="module")
def child(lib, tmp_path_factory):
    if not shutil.which("gcc") or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime_api.h")):
        pytest.skip("gcc and the CUDA headers are needed")
    so = str(tmp_path_factory.mktemp("fake") / "cudart.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-w", "-I" + CUDA_INCLUDE, "-o", so,
                    os.path.join(HERE, "fake", "cudart.c"), "-lpthread"], check=True)

    def call(code):
        env = dict(os.environ, LD_PRELOAD=so, PYTHONPATH=os.path.dirname(HERE))
        r = subprocess.run([sys.executable, "-c", PREAMBLE + code], env=env, capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stdout + r.stderr

    return call


def test_short_runs_take_no_second_array(child):
    """Fewer than four steps left, also after a leading beta step, cannot use it."""
    child("""
with solver() as s:
    held = s.info()["device_bytes"]
    assert [run(s, n) for n in (2, 3, 4, 1)] == [2, 3, 4, 1]   # 4: beta first, three left
    assert s.info()["device_bytes"] == held
    assert run(s, 8) == 4                                       # pairs
    assert s.info()["device_bytes"] > 1.9 * held
""")


def test_every_domain_of_a_batch_reports_an_expired_wait_once(child):
    """One launch steps all domains, so its failure is each one's."""
    child("""
def status(f, *a):
    try: f(*a)
    except LbmError as e: return e.status
    return 0
with batch((8, 8, 8), 4) as b:
    v = [b.domain(i) for i in range(4)]
    b.run(2)
    assert lib.lbm_selftest_bounded_wait(v[0]._h, 1000) == TIMEOUT      # raises the batch's flag
    assert status(v[1].getDensities) == TIMEOUT and status(v[1].getDensities) == 0
    assert lib.lbm_synchronize(v[2]._h) == TIMEOUT and status(v[2].getVelocities) == 0
    assert lib.lbm_selftest_bounded_wait(v[2]._h, 1000) == TIMEOUT
    assert [status(x.reduce) for x in v] == [TIMEOUT, TIMEOUT, 0, TIMEOUT]
    assert [status(x.reduce) for x in v] == [0] * 4
""")


@pytest.mark.parametrize("packed", [True, False])
def test_failed_copy_does_not_hide_an_expired_wait(child, packed):
    """The flag comes with the fields; a getter that fails after computing them leaves it to the next one."""
    child(f"packed = {packed}" + """
n = (20, 14, 11)
with solver(n) as s:
    err = []
    def steps_fail(name, args):  # the step kernel's work ends with its flag set
        if err and b"beta" in name: C.c_int.from_address(err[0]).value = 4
        if b"compute_macros" in name and not err:  # (..., err, host_err)
            err.append(C.c_void_p.from_address(args[6]).value)
    watch(steps_fail)
    s.getDensities()
    s.run(2)
    if not packed: fake.fake_memory(0)
    status = []
    for i in range(4):  # the runtime keeps a failed copy's error for the next launch to return
        fake.fake_fail_copies(1 if i == 0 else 0)
        try: s.getVelocities(); status.append(0)
        except LbmError as e: status.append(e.status)
    assert status == [3, 3, TIMEOUT, 0], status
""")


@pytest.mark.parametrize("at", [1, 2, 4])
def test_failed_pair_launch_leaves_a_batch_at_its_last_whole_step(child, at):
    """After the first of two passes the state is in the second pool only: the step counter counts both or none, and
    the domains stay at the batch's time level."""
    child(f"at = {at}" + """
with batch() as b:
    b.run(1)
    fake.fake_fail_launch(b"pair_step", at)
    try: b.run(17); status = 0
    except LbmError as e: status = e.status
    done = 2 + (at - 1) // 2 * 4
    assert status == 3 and b.info()["step_counter"] == done
    assert [b.domain(i).info()["step_counter"] for i in (0, 75)] == [done] * 2
    assert run(b, 8) == 4 and b.info()["step_counter"] == done + 8
""")


def test_second_pool_is_not_given_up_between_launches(child):
    """A domain's getter on another thread runs out of memory while the batch queues its passes: the pool they write to
    must be there until they are queued."""
    child("""
with batch() as b:
    v = b.domain(3)
    assert run(b, 4) == 2
    used, bad, reached = fake.fake_used(), [], threading.Event()
    def launch(name, args):
        if b"pair_step" not in name: return
        reached.set()
        time.sleep(0.05)
        # (map, domain, step_base, step_off, work, err); work ends with domains, domain_of, maps, out
        at = args[4]
        ptrs = [C.c_void_p.from_address(at + o).value for o in (24, 32, 40, 48)]
        if not all(fake.fake_live(p) for p in ptrs): bad.append(ptrs)
    watch(launch)
    fake.fake_memory(used)                                      # the getter's fields need the second pool's memory
    def get():
        reached.wait()
        v.getDensities()
    t = threading.Thread(target=get)
    t.start()
    assert run(b, 16) == 8
    t.join()
    assert not bad
    fake.fake_on_launch(None)
    assert fake.fake_used() < used                              # it has been given up
    assert run(b, 4) == 4
""")


@pytest.mark.parametrize("other", ["solver", "batch", "server", "fields", "autotune"])
def test_second_arrays_go_to_whoever_needs_the_memory(child, other):
    """What could be made before runs took second arrays can still be made after them."""
    child(f"other = {other!r}" + """
with solver() as a, batch() as b:
    half = a.info()["device_bytes"], b.info()["device_bytes"]
    assert run(a, 8) == 4 and run(b, 8) == 4
    both = a.info()["device_bytes"], b.info()["device_bytes"]
    assert both[0] > 1.9 * half[0] and both[1] > 1.5 * half[1]
    with solver((250, 256, 256)) as c:
        assert run(c, 4) == 2
        if other == "solver":
            fake.fake_memory(fake.fake_used() + 200 * MB)
            d = solver()
        elif other == "batch":
            fake.fake_memory(fake.fake_used() + 200 * MB)
            d = batch((64, 64, 60), 100)
        elif other == "server":
            fake.fake_memory(fake.fake_used() + 200 * MB)
            d = LbmServer(budget_bytes=2 * GB, storage="f16sr")
        elif other == "fields":
            fake.fake_memory(fake.fake_used())
            a.getDensities(out=np.empty((256, 256, 256), np.float32))
            d = None
        else:
            fake.fake_memory(fake.fake_used())
            c.autotune(1)
            d = None
        held = a.info()["device_bytes"] + b.info()["device_bytes"] + c.info()["device_bytes"]
        fake.fake_memory(1 << 40)
        if d: d.close()
        n = run(a, 8) + run(b, 8) + run(c, 8)
        assert 12 < n <= 24 and held < 2 * (half[0] + half[1] + half[0])
assert fake.fake_used() == 0
""")


def test_memory_that_is_nobodys_second_array_still_runs_out(child):
    child("""
with solver() as a:
    run(a, 8)
    fake.fake_memory(fake.fake_used() + 200 * MB)
    for make in (lambda: solver((512, 512, 256)), lambda: batch((64, 64, 64), 300),
                 lambda: LbmServer(budget_bytes=6 * GB, storage="f16sr")):
        try: make(); status = 0
        except LbmError as e: status = e.status
        assert status in (4, 8), status
    assert run(a, 8) == 8
""")


def test_chosen_variant_gives_the_second_array_back(child):
    child("""
for s in (solver(), batch()):
    held, used = s.info()["device_bytes"], fake.fake_used()
    assert run(s, 8) == 4 and s.info()["device_bytes"] > held
    s.set_fast_variant(s.info()["fast_variant"])
    assert s.info()["device_bytes"] == held and fake.fake_used() == used
    assert run(s, 8) == 8
    s.close()
""")


@pytest.mark.parametrize("share,pairs", [(3.9, False), (4.1, True)])
def test_second_array_takes_at_most_a_quarter_of_the_free_memory(child, share, pairs):
    child(f"share, pairs = {share}, {pairs}" + """
for make in (solver, batch):
    with make() as s:
        pop = 19 * s.info()["slot_stride"] * 4 if make is solver else 76 * 19 * s.domain(0).info()["slot_stride"] * 4
        fake.fake_memory(fake.fake_used() + int(share * pop))
        assert run(s, 8) == (4 if pairs else 8)
        fake.fake_memory(1 << 40)
        assert run(s, 8) == (4 if pairs else 8)    # refused for good
""")


def test_capturing_stream_takes_single_steps_and_no_memory(child):
    child("""
for make in (solver, batch):
    with make() as s:
        used = fake.fake_used()
        fake.fake_capturing(0x1000)
        before = kernel_launches()
        s.run(8, stream=0x1000)
        assert kernel_launches() - before == 8 and fake.fake_used() == used
        assert run(s, 8) == 4
""")


def test_memory_is_taken_without_breaking_a_capture_elsewhere(child):
    """Runs and the populations' getter took no memory before they took two steps a pass or packed: they still work
    beside a capture in global mode on another stream."""
    child("""
st = 0x2000
for make in (solver, batch):
    with make() as s, solver((40, 30, 20)) as t:
        fake.fake_capture_elsewhere(1)
        before = kernel_launches()
        s.run(8, stream=st)
        assert kernel_launches() - before == 4 and not fake.fake_capture_broken()
        out = np.empty((19, 20, 30, 40), np.float32)
        assert lib.lbm_get_density_distributions(t._h, None, None, out.ctypes.data, st) == 0
        s.set_fast_variant(s.info()["fast_variant"]) if make is solver else None
        assert not fake.fake_capture_broken()
        fake.fake_capture_elsewhere(0)
""")


def test_batch_without_room_for_row_padding_keeps_its_narrow_rows(child):
    """Rows are padded to what two steps a pass need only where those pay and the padded pool fits."""
    child("""
def pool(b, n, count):
    return count * 19 * 4 * b.domain(0).info()["slot_stride"]
for n, count, rows in (((2, 900, 900), 4, (6, 6)), ((64, 64, 64), 76, (68, 68)), ((65, 64, 64), 76, (72, 70))):
    with batch(n, count) as b:
        assert b.domain(0).info()["row_pitch"] == rows[0], b.domain(0).info()["row_pitch"]
        assert run(b, 8) == (8 if rows[0] == 6 else 4)
    with batch(n, count) as b:
        wide, rest = pool(b, n, count), b.info()["device_bytes"] - pool(b, n, count)
    if rows[0] == rows[1]: continue
    assert wide * rows[1] // rows[0] + rest < wide - 1
    fake.fake_memory(wide - 1)
    with batch(n, count) as b:
        assert b.domain(0).info()["row_pitch"] == rows[1]
        assert [b.domain(i).info()["row_pitch"] for i in (1, count - 1)] == [rows[1]] * 2
        fake.fake_memory(1 << 40)
        assert run(b, 8) == 8
""")


def test_info_does_not_wait_for_a_run(child):
    """A thread that watches another's run gets its answer while the launches are being queued."""
    child("""
for make in (solver, batch):
    with make() as s:
        run(s, 4)
        reached, times = threading.Event(), []
        def launch(name, args):
            if b"pair_step" in name:
                reached.set()
                time.sleep(0.1)
        watch(launch)
        def look():
            reached.wait()
            t = time.perf_counter()
            s.info()
            times.append(time.perf_counter() - t)
        t = threading.Thread(target=look)
        t.start()
        s.run(20)
        t.join()
        fake.fake_on_launch(None)
        assert times[0] < 0.05, times
""")


@pytest.mark.parametrize("kernel", ["alpha_fast", "beta_fast_direct", "pair_step", "batch_step"])
def test_failed_launch_is_reported_once(child, kernel):
    """The runtime keeps a launch's error until it is asked for: the call that failed takes it away, so that the next
    one does not report it again."""
    child(f"kernel = {kernel!r}.encode()" + """
with (batch() if kernel == b"batch_step" else solver()) as s:
    v = s.domain(3) if kernel == b"batch_step" else s
    if kernel != b"pair_step": s.set_fast_variant(s.info()["fast_variant"])
    run(s, 1 if kernel == b"beta_fast_direct" else 4)
    v.getDensities((1, 1, 1), (4, 4, 4))                        # the fields' memory is there
    fake.fake_fail_launch(kernel, 1)
    try: s.run(4); status = 0
    except LbmError as e: status = e.status
    assert status == 3
    s.run(1)
    v.getDensities((1, 1, 1), (4, 4, 4))
""")

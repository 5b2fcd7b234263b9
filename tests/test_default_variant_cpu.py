"""Default launch variants of the 16-bit storages on short rows, each side of the
borders (the cubes' borders are held by test_gpu_default_variant.py), on the
stand-in for the CUDA runtime; the results of every variant are held by the
parity tests."""
import pytest

from test_host_paths_cpu import child  # noqa: F401

CASES = [((25, 76, 76), 6), ((9, 103, 102), 6),  # 304 and 306 blocks of two cells a thread
         ((25, 80, 80), 8), ((30, 71, 70), 8), ((10, 122, 122), 8), ((13, 106, 105), 8), ((13, 111, 110), 8), ((9, 133, 133), 8),
         ((32, 70, 70), 6), ((11, 213, 213), 8),  # 83 MB: in L2
         ((11, 302, 301), 20), ((9, 333, 333), 20), ((12, 393, 392), 20), ((13, 196, 196), 8), ((13, 340, 339), 20), ((16, 256, 256), 20), ((8, 400, 400), 23),
         ((17, 297, 297), 23), ((26, 267, 266), 20), ((28, 215, 215), 23),  # 115 MB
         ((28, 257, 257), 20), ((29, 253, 252), 23), ((41, 212, 212), 23)]


@pytest.mark.parametrize("storage", ["f16s", "bf16s", "f16sr"])
def test_default_variant_of_short_rows(child, storage):  # noqa: F811
    child(f"""
for n, want in {CASES!r}:
    with solver(n, {storage!r}) as s:
        assert s.info()["fast_variant"] == want, (n, s.info()["fast_variant"])
""")


@pytest.mark.parametrize("storage,n,count,variant", [("f32", (20, 20, 20), 10, 13), ("f32", (64, 64, 64), 2, 14),
                                                     ("f64", (64, 64, 64), 4, 13), ("f64", (64, 64, 64), 5, 14),
                                                     ("f16sr", (20, 20, 20), 10, 22), ("f16sr", (64, 64, 64), 9, 22)])
def test_default_variant_of_batches(child, storage, n, count, variant):  # noqa: F811
    child(f"""
with batch({n}, {count}, {storage!r}) as b:
    assert b.info()["fast_variant"] == {variant}, b.info()["fast_variant"]
""")

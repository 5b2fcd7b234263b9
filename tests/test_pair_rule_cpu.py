"""When lbm_run takes two steps a pass (pair_step_pays), on the stand-in for the
CUDA runtime: boxes that pairs were measured to make slower keep single steps,
ordinary ones take pairs."""
import pytest

from test_host_paths_cpu import child  # noqa: F401

SLOWER = [("f16sr", (61, 63, 453)), ("f16sr", (291, 129, 161)), ("f16sr", (429, 203, 81)), ("f16sr", (441, 136, 66)),
          ("f16sr", (223, 79, 1291)), ("f32", (37, 157, 177)), ("f32", (39, 26, 963)), ("f32", (84, 120, 112)),
          ("bf16s", (447, 30, 149)), ("bf16s", (58, 218, 134)), ("bf16s", (143, 247, 337)), ("f16s", (58, 93, 305))]
FASTER = [("f32", (128, 128, 128)), ("f16sr", (128, 128, 128)), ("f32", (193, 200, 187)), ("f32", (384, 384, 384)), ("f16s", (160, 160, 160)),
          ("bf16s", (256, 256, 256)), ("f16sr", (192, 192, 192)), ("f16sr", (512, 512, 512)), ("f32", (61, 311, 567)),
          ("f16sr", (447, 300, 200))]


@pytest.mark.parametrize("storage,n,launches", [(*c, 8) for c in SLOWER] + [(*c, 4) for c in FASTER])
def test_pairs_only_where_they_are_faster(child, storage, n, launches):  # noqa: F811
    child(f"""
with solver({n}, {storage!r}) as s:
    got = run(s, 8)
assert got == {launches}, got
""")

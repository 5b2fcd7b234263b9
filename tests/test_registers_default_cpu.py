"""Register budgets, as test_registers_cpu.py checks them, of the kernels that
run by default and are not in its list: two steps a pass (single domains and
FP32 batches), FP64 with integer products, the 16-bit storages' variants for
small domains, FP32 and FP64 batches."""
import shutil
import subprocess
from concurrent.futures import ThreadPoolExecutor

import pytest

from test_registers_cpu import ptxas_report

# (translation unit, kernel, most registers or None, most spilled bytes): blocks of pair_step are alone on their SM, 672
# threads at 96 registers or 768 at 80
BUDGETS = [
    ("lbm_pair.cu", "pair_step<lbm::F32, 64, 8, 4, false>", 96, 0),
    ("lbm_pair.cu", "pair_step<lbm::F32, 64, 8, 4, true>", 96, 0),
    ("lbm_pair.cu", "pair_step<lbm::F16S, 64, 10, 5, false>", 80, 0),
    ("lbm_pair.cu", "pair_step<lbm::BF16S, 64, 10, 5, false>", 80, 0),
    ("lbm_pair.cu", "pair_step<lbm::F16SR, 64, 10, 5, false>", 80, 0),
    ("fast_f32.cu", "batch_step<lbm::F32, 2, 128, 4, true, 2>", 128, 48),
    ("fast_f32.cu", "batch_step<lbm::F32, 2, 128, 4, false, 2>", 128, 0),
    ("fast_f64.cu", "alpha_fast<lbm::F64, 1, 64, 8>", 128, 0),
    ("fast_f64.cu", "beta_fast_direct<lbm::F64, 1, 64, 8>", 128, 0),
    ("fast_f32.cu", "batch_step<lbm::F32, 2, 64, 8, true, 2>", 128, 48),
    ("fast_f32.cu", "batch_step<lbm::F32, 2, 64, 8, false, 2>", 128, 0),
    ("fast_f64.cu", "batch_step<lbm::F64, 1, 64, 8, true, 2>", 128, 0),
    ("fast_f64.cu", "batch_step<lbm::F64, 1, 64, 8, false, 2>", 128, 0),
    ("fast_f64.cu", "batch_step<lbm::F64, 1, 128, 4, true, 2>", 128, 0),
    ("fast_f64.cu", "batch_step<lbm::F64, 1, 128, 4, false, 2>", 128, 0),
    ("fast_f16sr.cu", "alpha_fast<lbm::F16SR, 2, 256, 2>", 128, 0),
    ("fast_f16sr.cu", "beta_fast<lbm::F16SR, 2, 256, 2>", 128, 0),
    ("fast_f16sr.cu", "alpha_fast<lbm::F16SR, 4, 64, 8>", 128, 0),
    ("fast_f16sr.cu", "beta_fast_blk<lbm::F16SR, 4, 64, 8>", 128, 6),
    ("fast_f16sr.cu", "beta_fast_pk<lbm::F16SR, 4, 64, 10, true>", 96, 16),
]


@pytest.mark.skipif(shutil.which("nvcc") is None or shutil.which("c++filt") is None,
                    reason="nvcc and c++filt are needed")
def test_kernels_that_run_by_default_fit_their_register_budgets(tmp_path):
    units = sorted({u for u, *_ in BUDGETS})
    with ThreadPoolExecutor(len(units)) as pool:
        reports = dict(zip(units, pool.map(lambda u: ptxas_report(u, str(tmp_path)), units)))
    for unit, kernel, max_regs, max_spill in BUDGETS:
        mangled = list(reports[unit])
        names = subprocess.run(["c++filt"], input="\n".join(mangled), capture_output=True, text=True,
                               check=True).stdout.splitlines()
        hits = [reports[unit][m] for m, n in zip(mangled, names) if n.split("(")[0] == "void lbm::" + kernel]
        assert len(hits) == 1, (unit, kernel, len(hits))
        assert hits[0][1] is not None and hits[0][1] <= max_spill and hits[0][0] <= max_regs, (kernel, hits[0])

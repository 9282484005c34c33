"""Integer products store through shared memory only: a kernel configuration whose
stages leave no room for it does not compile (the row-wise store would take its
sums for floats)."""
import os
import subprocess

import pytest

from ferray_b200 import build

SRC = """
#include "tc_gemm2.cuh"
using namespace fg;
using Cfg = Tc2Cfg<KIND_I8, 256, %d, 1, 1, 1, 1, EPI_I32>;
const void* kernel = reinterpret_cast<const void*>(tc_gemm2_kernel<Cfg>);
"""


@pytest.mark.parametrize("stages,compiles", [(6, True), (7, False)])
def test_stages_leave_room_for_the_stores(tmp_path, stages, compiles):
    src = tmp_path / "cfg.cu"
    src.write_text(SRC % stages)
    r = subprocess.run([build.NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O0", "-I" + build.CSRC,
                        "-I" + os.path.join(build.ROOT, "include"), "-c", str(src), "-o", os.devnull],
                       capture_output=True, text=True)
    assert (r.returncode == 0) == compiles, r.stderr
    if not compiles:
        assert "integer outputs leave through shared memory only" in r.stderr

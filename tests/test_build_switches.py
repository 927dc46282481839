"""Build switches that the kernels' shared memory and waits depend on: values
that they do not allow are refused when the library is compiled."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cup-cfd_b200", "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.parametrize("header,switch,fine", [
    ("kernels_pf.cuh", "CUPCFD_STAGE_FROM=4", True),
    ("kernels_pf.cuh", "CUPCFD_STAGE_FROM=3", False),   # the last face's copy would never be waited for
    ("ordered_sum.cuh", "CUPCFD_OS_T=256", True),
    ("ordered_sum.cuh", "CUPCFD_OS_T=96", False),
    ("ordered_sum.cuh", "CUPCFD_OS_T=4096", False),
    ("ordered_sum.cuh", "CUPCFD_OS_FIRST=0", False),
])
def test_switch(tmp_path, header, switch, fine):
    if not os.path.exists(NVCC):
        pytest.skip("no nvcc")
    # naming a member makes the compiler complete the staging buffer's type
    use = "static_assert(sizeof(cupcfd_gpu::FwdMadjStage<64>) > 0, \"\");" if header == "kernels_pf.cuh" else ""
    (tmp_path / "t.cu").write_text(f'#include "{header}"\n{use}\n')
    r = subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", CSRC, "-I",
                        os.path.join(CSRC, "..", "..", "include"), f"-D{switch}", "-c", str(tmp_path / "t.cu"), "-o",
                        str(tmp_path / "t.o")], capture_output=True, text=True)
    assert (r.returncode == 0) == fine, r.stderr
    assert fine or "static assertion failed" in r.stderr or "static_assert" in r.stderr, r.stderr

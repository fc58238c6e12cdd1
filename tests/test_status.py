"""The factorization's time-outs in words (host code only)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")

SRC = """
#include "pgpu_common.cuh"
#include <cstdio>
int main() {
    for (int k = 0; k < 4; k++) {
        pgpu::Status st = {};
        if (k == 1) st.timeout = 3;
        if (k == 2) st.panel_timeout = 5;
        if (k == 3) st.panel_timeout = 7, st.drain_timeout = 1;
        printf("[%s]", pgpu::status_timeouts(st).c_str());
    }
}
"""


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
def test_block_row_timeouts_are_reported_apart(tmp_path):
    """A wait that gives up in the diagonal blocks is not blamed on the tensor-core kernels."""
    src, exe = tmp_path / "status.cu", tmp_path / "status"
    src.write_text(SRC)
    subprocess.check_call([NVCC, "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a",
                           "-I", os.path.join(ROOT, "pastix_b200", "csrc"), "-o", str(exe), str(src)])
    none, tc, panel, both = subprocess.check_output([str(exe)], text=True)[1:-1].split("][")
    assert none == ""
    assert "3 CTAs' tensor-core" in tc and "diagonal" not in tc
    assert "5 CTAs" in panel and "diagonal blocks" in panel and "tensor-core" not in panel
    assert "7 CTAs" in both and "undefined" in both

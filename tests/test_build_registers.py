"""What the compiler reports for kernels whose comments state it."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.join(os.path.dirname(__file__), "..")


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc")
def test_csr_row_writer_does_not_spill(tmp_path):
    r = subprocess.run(
        ["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
         "-I", os.path.join(ROOT, "include"), "--expt-relaxed-constexpr", "-Xptxas", "-v", "-c",
         "-o", str(tmp_path / "csr.o"), os.path.join(ROOT, "cuppa-public_b200", "csrc", "pa_csr.cu")],
        capture_output=True, text=True, check=True)
    report = re.findall(r"Function properties for (\S*rows_kernel\S*)\s+.*?(\d+) bytes spill stores, "
                        r"(\d+) bytes spill loads", r.stdout + r.stderr)
    assert len(report) == 2   # both id widths
    assert all(stores == loads == "0" for _, stores, loads in report), report

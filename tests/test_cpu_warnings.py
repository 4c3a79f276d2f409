"""The kernel sources compile without a warning: nvcc's are about code that
nothing reaches, or, as for a __shared__ variable with initialisers, about what
the device compiler does not do."""
import concurrent.futures as cf
import glob
import os
import shutil
import subprocess

import pytest

from turbins_gb300 import build as B


def test_sources_compile_without_warnings(tmp_path):
    if not (shutil.which("nvcc") or os.path.exists("/usr/local/cuda/bin/nvcc")):
        pytest.skip("no nvcc")

    def comp(src):
        # the front end's warnings need no optimisation
        cmd = [B.nvcc()] + B.ARCH + ["-O0", "-Xptxas", "-O0", "-std=c++17", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC",
                                     "-c", src, "-o", str(tmp_path / (os.path.basename(src) + ".o"))]
        r = subprocess.run(cmd, capture_output=True, text=True)
        return src, r.returncode, r.stdout + r.stderr

    with cf.ThreadPoolExecutor(max_workers=8) as ex:
        for src, rc, log in ex.map(comp, sorted(glob.glob(os.path.join(B.CSRC, "*.cu")))):
            assert rc == 0, log
            assert "warning" not in log, (src, log)

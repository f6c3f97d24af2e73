"""The MMA update kernel is instantiated for one to five constraints; with five, a reduction carries
more values than a 32-bit mask of the maxima has bits.  The compiler says so: no warning may come up."""
import os
import subprocess

import pytest

from robustoptspline3d_b200 import build as B


def test_mma_kernels_compile_without_warnings(tmp_path):
    if not os.path.exists(B.NVCC):
        pytest.skip("no nvcc")
    cmd = [B.NVCC] + B.ARCH + B.FLAGS + ["-Werror", "all-warnings", "-ptx", "-o", str(tmp_path / "mma.out"),
                                         os.path.join(B.SRC, "mma.cu")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

"""A look-back wait of the radix passes that runs out is reported, and nothing is written on the
strength of what that pass left behind (radix_wait.cu, built with a bound of 4,096 polls)."""
import subprocess
from pathlib import Path

import pytest

from psc import _build

pytestmark = pytest.mark.gpu


def test_given_up_wait_ends_the_sort(cuda_device, tmp_path):
    exe = tmp_path / "radix_wait"
    src = Path(__file__).resolve().parent / "radix_wait.cu"
    _build._run([_build.NVCC, *_build.ARCH, *_build.NVCC_FLAGS, "-DPSC_RS_SPIN=4096",
                 f"-I{_build.CSRC}", str(src), str(_build.BUILD / "graph.o"), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60, check=True).stdout
    assert out.split() == ["failed", "1", "written", "0", "offsets", "0", "error", "0"]

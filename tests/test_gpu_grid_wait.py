"""Barriers of the resident launches: a wait that runs out ends the launch with its flag set, and
the bound that the library is built with is far above the longest step of a solve (grid_wait.cu)."""
import subprocess
from pathlib import Path

import pytest

from psc import _build

pytestmark = pytest.mark.gpu


def test_bound(cuda_device, tmp_path):
    exe, src = tmp_path / "grid_wait", Path(__file__).resolve().parent / "grid_wait.cu"
    _build._run([_build.NVCC, *_build.ARCH, *_build.NVCC_FLAGS, "-DPSC_GRID_SPIN=262144u",
                 f"-I{_build.CSRC}", str(src), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60, check=True).stdout
    w = out.split()
    assert w[0] == "gave_up" and w[1] == w[3] and w[4:6] == ["failed", "1"], out
    assert 25 < float(w[7]) < 400, out

"""The fused step (auto's choice for most grids) in the index-checked library: its
source carries the checks, and its cases -- tile and chunk edges, every boundary
letter, lossy media, mu arrays, current boxes on faces, slabs that are absent,
narrow and wider than a box copy -- pass with them, so no index of theirs leaves
its array (test_gpu_checked does the same for the pair and the serving kernel)."""
import os
import subprocess
import sys

import pytest

from emopt_b200 import build
from helpers import ROOT


def test_the_stepping_sources_carry_the_checks():
    assert {"vec_kernels.cu", "zmarch_kernels.cu", "serve_kernels.cu"} <= set(build.CHECKED_SOURCES)


@pytest.mark.gpu
def test_fused_cases_pass_with_index_checks():
    assert os.path.exists(build.CHECKED), "build the checked library first (python -m emopt_b200.build)"
    cmd = [sys.executable, "-m", "pytest", "-q", "-x", "-m", "gpu", "-p", "no:cacheprovider", "tests/test_gpu_march.py",
           "tests/test_gpu_mixed_mu.py", "tests/test_gpu_auto_kernel.py"]
    out = subprocess.run(cmd, cwd=ROOT, env=dict(os.environ, EMOPT_B200_LIB=build.CHECKED), capture_output=True,
                         text=True, timeout=1200)
    print(out.stdout[-3000:], out.stderr[-2000:])
    assert out.returncode == 0 and " passed" in out.stdout

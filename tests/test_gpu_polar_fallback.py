"""The rotation matrix where the cooperative launch is not to be had: step by step for whole tiles, on the host for other widths."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("dim,m", [(40, 10), (48, 12), (123, 41)])
def test_rotation_without_the_cooperative_launch(dim, m):
    code = f"import oracle; from tests.test_gpu_polar import test_rotation_is_the_polar_factor as t; t(oracle, {dim}, {m})"
    subprocess.run([sys.executable, "-c", code], cwd=ROOT, env={**os.environ, "VQB_POLAR_STEPWISE": "1"}, check=True, timeout=300)

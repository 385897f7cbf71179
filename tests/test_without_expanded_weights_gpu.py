"""The kernels that serve when weights could not be expanded to fp16 (no room on the device): the tests of the batched
products, of the SwiGLU forms and of whole models, in a process that makes no expanded copies."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
TESTS = ["test_ops_gpu.py::test_matmul_stores", "test_swiglu_gpu.py", "test_lfm2_gpu.py", "test_qwen35_gpu.py"]


def test_products_without_expanded_weights():
    ran = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-m", "gpu", "-p", "no:cacheprovider"] + [os.path.join(HERE, t) for t in TESTS],
                         env=dict(os.environ, BOBCAT_NO_HALF_MATMUL="1"), cwd=os.path.dirname(HERE), capture_output=True, text=True, timeout=900)
    assert ran.returncode == 0, ran.stdout[-4000:] + ran.stderr[-2000:]
    assert " passed" in ran.stdout

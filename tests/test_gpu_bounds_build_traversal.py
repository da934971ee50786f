"""The traversal and adjoint suites against the index-checked build, whose
kernels check their stacks, queues and lists in shared memory too (see
test_gpu_bounds_build.py)."""
import os
import subprocess
import sys

import pytest
import torch

from test_gpu_bounds_build import LIB, ROOT

pytestmark = pytest.mark.gpu

SUITES = ["test_gpu_packets_tiles.py", "test_gpu_packet_stack.py", "test_gpu_packet_margins.py",
          "test_gpu_adjoint_cutoff.py", "test_gpu_adjoint_rounding.py", "test_gpu_tree_edges.py"]


@pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA device")
def test_traversal_suites_pass_under_index_checks():
    if not os.path.exists(LIB):
        pytest.fail(f"{LIB} is missing: build it with `make -C diff-triangle-tracer_b200 bounds`")
    env = dict(os.environ, TRITRACER_LIB=LIB)
    cmd = [sys.executable, "-m", "pytest", "-q", "-x", "-m", "gpu", "-p", "no:cacheprovider"]
    cmd += [os.path.join(ROOT, "tests", s) for s in SUITES]
    res = subprocess.run(cmd, cwd=ROOT, env=env, capture_output=True, text=True, timeout=1200)
    assert res.returncode == 0, res.stdout[-3000:] + res.stderr[-2000:]
    assert "passed" in res.stdout

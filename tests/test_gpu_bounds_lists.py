"""The bounds-check build on the list passes at their edges, the octree and the
adjoint: the tests of those run again in a child process that loads it, and
report no index out of range."""
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.mark.gpu
def test_bounds_check_build_runs_the_list_tests_clean():
    lib = os.path.join(ROOT, "meshtrex_b200", "libmeshtrex_b200_check.so")
    assert os.path.exists(lib), "build it with `make -C meshtrex_b200/csrc check`"
    files = ["test_gpu_cell_lists.py", "test_gpu_octree_tiles.py", "test_gpu_adjoint_dense.py",
             "test_gpu_adjoint_faces.py", "test_gpu_block_shares.py"]
    r = subprocess.run([sys.executable, "-m", "pytest", "-x", "-q", "-m", "gpu", *(os.path.join(HERE, f) for f in files)],
                       capture_output=True, text=True, env=dict(os.environ, MESHTREX_B200_LIB=lib), cwd=ROOT, timeout=900)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]

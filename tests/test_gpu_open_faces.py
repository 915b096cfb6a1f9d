"""The device check that no defined cell lies next to an unallocated brick
holds in bricks at remapping boundaries too: an error for every face past which
the grid goes on, none at a mirroring wall."""
import os
import subprocess

import pytest

from viennals_b200 import BoundaryConditionEnum as BC

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_faces_of_bricks_at_boundaries(tmp_path):
    exe = str(tmp_path / "open_faces")
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.check_call([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17",
                           "--expt-relaxed-constexpr", "-I",
                           os.path.join(ROOT, "viennals_b200", "csrc"),
                           os.path.join(ROOT, "tests", "cpp", "open_faces.cu"), "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0
    rows = [tuple(map(int, r.split())) for r in out.stdout.splitlines()]
    assert len(rows) == 5 * 6 * 2
    for bc, face, allocated, err in rows:
        lower = face % 2 == 0
        mirror = (bc == BC.REFLECTIVE_BOUNDARY or (bc == BC.POS_INFINITE_BOUNDARY and lower) or
                  (bc == BC.NEG_INFINITE_BOUNDARY and not lower))
        assert err == (0 if allocated or mirror else 64), (bc, face, allocated)

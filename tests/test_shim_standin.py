"""The eigensolve_lanczos drop-in builds without a NEMO-3D tree.

``tests/shim/build_shim.sh`` without the reference's headers compiles against
tests/shim/standin, so that tests/test_gpu_shim.py has a library to call.
Bars: the recipe succeeds without diagnostics and the library exports the
entry point; where the tree is present tests/test_shim.py covers the build.
"""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
REF = os.environ.get("NEMO3D_SRC", "/root/reference/NEMO_3D")


def test_shim_builds_without_the_reference_tree():
    if os.path.isdir(REF):
        pytest.skip("reference headers present")
    env = {k: v for k, v in os.environ.items() if k != "NEMO3D_SRC"}
    p = subprocess.run(["sh", os.path.join(HERE, "shim", "build_shim.sh")], env=env,
                       capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr
    assert "warning" not in p.stderr and "error" not in p.stderr, p.stderr
    lib = ctypes.CDLL(os.path.join(HERE, "shim", "_build", "libtbgpu_shim.so"))
    assert hasattr(lib, "eigensolve_lanczos")

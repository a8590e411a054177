"""The build description, without building: the library needs CUDA alone, the Python binding is built where torch is found."""
import os
import subprocess
import sys

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ops-cv_b200", "csrc")


def plan(*args):
    """What make would run if nothing were built yet."""
    run = subprocess.run(["make", "-n", "-B", "-C", CSRC, *args], capture_output=True, text=True)
    assert run.returncode == 0, run.stderr
    return run.stdout


def test_library_builds_without_python_or_torch():
    for args in (("PYTHON=/nonexistent/python",), ("lib",), ("lib", "PYTHON=/nonexistent/python")):
        out = plan(*args)
        assert "libopscv_b200.so" in out and "_opscv_torch.so" not in out and "py_binding" not in out


def test_binding_is_built_where_torch_is_found():
    out = plan("PYTHON=" + sys.executable)
    assert "libopscv_b200.so" in out and "_opscv_torch.so" in out

"""What the host's make targets need: the C++ library nothing of Python, the extension module Python's headers."""
import os
import subprocess

HOST = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "x-deeplearning_b200", "host")


def _commands(*targets):
    """What make would run for these targets if nothing was built, with no Python to ask."""
    p = subprocess.run(["make", "-n", "-B", "-C", HOST, "PYTHON=/nonexistent/python3", *targets], capture_output=True, text=True)
    return p.stdout + p.stderr


def test_the_library_is_built_without_python():
    out = _commands("all")
    assert "libblaze_b200.so" in out and "xb_binding" not in out and "nonexistent" not in out


def test_the_extension_module_is_a_target_of_its_own():
    out = _commands("python")
    assert "xb_binding.so" in out and "libblaze_b200.so" not in out

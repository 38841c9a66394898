"""State that a context or the process keeps between calls, as compiled checks
of the library's host sources against CUDA calls that the checks define."""
import os

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _host_check(tmp_path, name, *sources):
    """Builds tests/host/<name>.cpp with library sources (CUDA calls that the check does not define stay unresolved)."""
    import shutil
    import subprocess
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host C++ compiler")
    exe = tmp_path / name
    inc = os.path.join(REPO, "vina-cuda_b200", "csrc")
    subprocess.run([gxx, "-std=c++17", "-O1", "-Wall", "-pthread", "-I", inc, "-I", "/usr/local/cuda/include",
                    os.path.join(REPO, "tests", "host", name + ".cpp"), *[os.path.join(inc, s) for s in sources],
                    "-Wl,--unresolved-symbols=ignore-all", "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


def test_host_stage_check(tmp_path):
    """The pinned stage when pinned memory is refused (a compiled host check)."""
    _host_check(tmp_path, "host_stage_check", "api.cpp", "tables.cpp")


def test_launch_settings_check(tmp_path):
    """The kernels' launch settings when several contexts set them (a compiled host check)."""
    _host_check(tmp_path, "launch_settings_check", "api.cpp", "tables.cpp")

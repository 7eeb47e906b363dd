"""Host-side decisions before a launch (tests/host_plan.cpp), on the CPU."""
import os
import shutil
import subprocess

import pytest

from test_host_kernels import HERE, ROOT, _cuda_include


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    cxx, inc = shutil.which("g++"), _cuda_include()
    if cxx is None or inc is None:
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path_factory.mktemp("hp") / "host_plan")
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "library_s_grand_gb300", "csrc"),
                    "-I", os.path.join(ROOT, "include"), "-I", inc,
                    os.path.join(HERE, "host_plan.cpp"), "-o", exe],
                   check=True, capture_output=True, text=True)
    return exe


def _run(exe, *args):
    p = subprocess.run([exe, *map(str, args)], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0, (p.returncode, p.stdout, p.stderr)
    return p.stdout.split()


def test_per_shot_buffer_layout(plan):
    _run(plan, "layout")


def test_rounds_go_on_while_shots_get_fewer(plan):
    _run(plan, "rounds")


def test_status_bits(plan):
    _run(plan, "status")


def test_every_entry_point_uses_the_same_rule():
    """No entry point tests the bits by itself: one that left the wait limit out returned 0."""
    for name in ("grand_host.cpp", "grand_engine.cpp", "grand_server.cpp", "grand_noalloc.cu"):
        with open(os.path.join(ROOT, "library_s_grand_gb300", "csrc", name), encoding="utf-8") as f:
            code = f.read()
        assert "status_code(" in code and "kStatusWaitLimit" not in code and "kStatusTamLimit" not in code, name

"""What the host shim queues, and when it may touch what a queued operation still reads: fsb_shim.cpp over a stand-in for the
CUDA runtime that runs queued operations as late as it may (tests/host_order.cpp)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    gxx = shutil.which("g++")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    if not gxx or not os.path.exists(os.path.join(cuda, "include", "cuda_runtime.h")):
        pytest.skip("no g++ or no CUDA toolkit on this machine")
    exe = str(tmp_path_factory.mktemp("host_order") / "host_order")
    cmd = [gxx, "-std=c++17", "-O1", "-Wall", "-I", os.path.join(cuda, "include"), os.path.join(ROOT, "tests", "host_order.cpp"),
           os.path.join(ROOT, "ferro_b200", "csrc", "fsb_shim.cpp"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


@pytest.mark.parametrize("args", [
    ("queued", 8), ("queued", 64), ("queued", 65), ("merged", 8), ("merged", 65),   # redraw, launch, redraw, launch, ... without waiting
    ("waited", 8), ("waited", 65),                                                  # ... after steps that were waited for
    ("replayed", 8), ("replayed", 64), ("replayed", 65),                            # a captured launch, replayed after redraws
    ("overlap",),                                                                   # mode 1 over histories in the id pool
    ("switched",),                                                                  # histories set on one stream, used on another
    ("drafts",),                                                                    # drafts of any 32-bit value
])
def test_host_order(driver, args):
    r = subprocess.run([driver, *map(str, args)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr

"""The streaming kernel's early bound under the softcap: a number that no cell of masked logits reaches, at or below the bound without
the softcap, and low enough that nothing below it can reach, after the softcap, what a logit at the bound does - for every cap that an engine
takes, the largest too, where four caps are more than a float holds."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_admit_of_a_softcap(tmp_path):
    import torch
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc on this machine")
    so = str(tmp_path / "libsoftcap_admit.so")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "-shared", "-cudart", "static",
                        os.path.join(ROOT, "tests", "softcap_admit.cu"), "-o", so], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(so)
    lib.softcap_admit_of.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_void_p]
    most = np.finfo(np.float32).max
    caps = np.array([0.5, 30.0, 1e6, 8e37, 8.5e37, 8.6e37, 1e38, most], np.float32)
    thrs = np.array([-most, -1e38, -200.0, -1.0, 0.0, 0.3, 25.0, 125.0, 1e30, most], np.float32)
    thr, cap = (np.ascontiguousarray(x.ravel()) for x in np.meshgrid(thrs, caps))
    dev = [torch.from_numpy(x).cuda() for x in (thr, cap)] + [torch.zeros(len(thr), device="cuda")]
    torch.cuda.synchronize()
    assert lib.softcap_admit_of(dev[0].data_ptr(), dev[1].data_ptr(), len(thr), dev[2].data_ptr()) == 0
    admit = dev[2].cpu().numpy()
    assert np.isfinite(admit).all(), list(zip(thr, cap, admit))
    assert (admit <= thr).all()

    def softcapped(x):
        return cap.astype(np.float64) * np.tanh(x.astype(np.float64) / cap.astype(np.float64))

    # (a bound of -FLT_MAX admits everything; the margin under the value at the bound is 2^-20 caps)
    assert ((admit == -most) | (softcapped(admit) <= softcapped(thr) - cap.astype(np.float64) * 2.0**-20)).all()

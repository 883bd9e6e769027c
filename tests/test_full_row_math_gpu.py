"""The full-vocabulary kernel's own division and exponential against the device's division and 80-bit exponentials.

Division: equal to the correctly rounded quotient, bit for bit.  Exponential of that quotient, in units of 2^-62: the
table's entries are off by at most 2^-52 of their value (an ulp of exp2), the last fused operation rounds by 2^-53, the
polynomial leaves out r^6 / 720 < 2^-54.6 (|r| <= ln 2 / 128) and all other roundings are below 2^-58; the conversion rounds to
a unit or less: |w - e| <= 1.75 * 2^-52 e + 1 unit."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def math(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc on this machine")
    so = str(tmp_path_factory.mktemp("math") / "libfull_row_math.so")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "-shared", "-cudart", "static",
                        os.path.join(ROOT, "tests", "full_row_math.cu"), "-o", so], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(so)
    lib.full_row_math.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_void_p, C.c_void_p]
    return lib


def arguments(kind, n, rng):
    if kind == "usual":       # temperatures that are asked for
        temp = rng.uniform(0.05, 2.0, n).astype(np.float32)
    elif kind == "any":       # all that a row of finite logits may have, denormal ones among them
        temp = (2.0 ** rng.uniform(-148, 119, n)).astype(np.float32)
    else:                     # significands at the ends of their range
        temp = ((1.0 + rng.choice([0, 1, 2, 2**22, 2**23 - 2, 2**23 - 1], n) * 2.0**-23) * 2.0 ** rng.integers(-20, 20, n)).astype(np.float32)
    diff = (-temp.astype(np.float64) * rng.choice([1e-6, 0.01, 1.0, 10.0, 45.0], n) * rng.random(n)).astype(np.float32)
    if kind == "edges":
        diff = -np.abs(diff.view(np.int32) & ~np.int32(0x7fffff) | rng.choice([0, 1, 2**22, 2**23 - 1], n).astype(np.int32)).view(np.float32)
        diff = -np.abs(diff)
    diff = np.maximum(diff, np.float32(-45.0) * temp)   # as the kernel cuts it
    diff[:3] = [0.0, -0.0, -np.float32(45.0) * temp[2]]
    return diff, temp


@pytest.mark.parametrize("kind", ["usual", "any", "edges"])
def test_division_and_exponential(math, kind):
    import torch
    n = 1 << 21
    diff, temp = arguments(kind, n, np.random.default_rng(len(kind)))
    assert np.isfinite(diff).all() and np.isfinite(temp).all() and (temp > 0).all() and (diff <= 0).all()
    dev = [torch.from_numpy(x).cuda() for x in (diff, temp)] + [torch.zeros(n, dtype=t, device="cuda") for t in (torch.float64, torch.float64, torch.int64)]
    torch.cuda.synchronize()
    assert math.full_row_math(dev[0].data_ptr(), dev[1].data_ptr(), n, *(x.data_ptr() for x in dev[2:])) == 0
    quotient, divided, weight = (x.cpu().numpy() for x in dev[2:])
    assert np.array_equal(quotient, divided) and np.array_equal(quotient, diff.astype(np.float64) / temp.astype(np.float64))
    exact = np.exp(quotient.astype(np.longdouble)) * np.longdouble(2.0) ** 62
    off = np.abs(weight.astype(np.longdouble) - exact)
    bound = exact * np.longdouble(1.75 * 2.0**-52) + 1
    worst = int(np.argmax(off / bound))
    print(kind, "largest error in units of the bound", float(off[worst] / bound[worst]))
    assert off[worst] <= bound[worst], (diff[worst], temp[worst], weight[worst], exact[worst])

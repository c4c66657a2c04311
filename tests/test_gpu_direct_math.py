"""The pair kernel's reciprocal (csrc/pme_direct_math.h) against CUDA's division."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

pytestmark = pytest.mark.gpu


def test_reciprocal_is_within_an_ulp(cuda, tmp_path):
    """Squared distances of 2^-30 to 2^40 A^2 with mantissas at random, at both ends and around the 20
    leading bits that the hardware's guess reads: the guess within 2^-19, the result within one ulp."""
    from gpu_recip_b200 import build
    lib = str(tmp_path / "direct_math.so")
    subprocess.run([build.nvcc()] + build.ARCH + ["-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I", build.CSRC,
                    os.path.join(ROOT, "tests", "cpp", "direct_math.cu"), "-o", lib], check=True)
    rng = np.random.default_rng(8)
    m = 1.0 + rng.random(400000)
    edge = 1.0 + np.concatenate([np.arange(64) * 2.0 ** -52, 1.0 - np.arange(1, 65) * 2.0 ** -53,
                                 (np.arange(2 ** 14) * 64 + rng.integers(0, 64, 2 ** 14)) * 2.0 ** -20,
                                 np.arange(2 ** 14) * 2.0 ** -14 + 2.0 ** -20 - 2.0 ** -52])
    x = np.concatenate([m * 2.0 ** rng.integers(-30, 41, m.size), edge, edge * 64.0])
    xd = cuda.from_numpy(x).cuda()
    out = [cuda.empty_like(xd) for _ in range(3)]
    rc = ctypes.CDLL(lib).reciprocal_run(ctypes.c_void_p(xd.data_ptr()), ctypes.c_int(x.size),
                                         *[ctypes.c_void_p(o.data_ptr()) for o in out])
    assert rc == 0
    guess, mine, division = (o.cpu().numpy() for o in out)
    assert np.array_equal(division, 1.0 / x)
    assert np.abs(guess).max() < 2.0 ** -19
    assert (np.abs(mine - division) <= np.spacing(division)).all()

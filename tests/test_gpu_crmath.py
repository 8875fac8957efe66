"""The device forms of gp_crmath.cuh (straight-line reciprocals and roots, CUDA's asinf
as the start of acos) against binary128 rounded once, compiled with the flags of the
FP64 unit and of the mixed unit, on the arguments of test_crmath.py; and the start
value's error, which the rounding test of acos_cr takes to be below 2^-21."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from gpluto_dev_b200 import build
from test_crmath import _acos_args, crm  # noqa: F401  (fixture)

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module", params=["fp64", "mixed"])
def dev(request, tmp_path_factory):
    so = str(tmp_path_factory.mktemp("crmath") / ("probe_%s.so" % request.param))
    flags = ["-fmad=false"] if request.param == "fp64" else build.MIXED_FP32
    subprocess.run([build.nvcc(), *build.ARCH, *build.BASE, *flags, "-shared",
                    os.path.join(HERE, "crmath_probe.cu"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    lib.crmath_probe.argtypes = [ctypes.c_void_p] * 2 + [ctypes.c_int] * 2

    def run(which, x):
        x = torch.as_tensor(x, dtype=torch.float64, device="cuda").contiguous()
        out = torch.empty_like(x)
        assert lib.crmath_probe(x.data_ptr(), out.data_ptr(), x.numel(), which) == 0
        return out.cpu().numpy()
    return run


def test_acos(dev, crm):  # noqa: F811
    rng = np.random.default_rng(21)
    tiny = 10.0 ** rng.uniform(-308, -8, 2000)
    x = np.concatenate([_acos_args(1_000_000, 1), tiny, -tiny])
    _, want = crm(0, x)
    bad = np.flatnonzero(dev(0, x) != want)
    assert bad.size == 0, (bad.size, x[bad[:5]])


@pytest.mark.parametrize("which", [1, 2])
def test_sin_cos(dev, crm, which):  # noqa: F811
    rng = np.random.default_rng(10 + which)
    x = np.concatenate([np.arccos(_acos_args(500_000, 2 + which)) / 3.0,
                        rng.uniform(0, 1.125, 500_000), np.arange(19) / 16.0,
                        10.0 ** rng.uniform(-300, 0, 1000), [0.0, 1.125]])
    x = x[(x >= 0) & (x <= 1.125)]
    _, want = crm(which, x)
    bad = np.flatnonzero(dev(which, x) != want)
    assert bad.size == 0, (bad.size, x[bad[:5]])


def test_start_of_acos(dev):
    """s = sqrt((1 -+ x)/2) >= 2^-27.5, or |x| <= 1/2; below 2^-28 acos only needs s to an
    absolute 2^-100 or so."""
    rng = np.random.default_rng(4)
    s = np.concatenate([rng.uniform(0, np.sqrt(0.5), 1 << 22), 2.0 ** rng.uniform(-28, 0, 1 << 20)])
    s = s[(s >= 2.0 ** -28) & (s <= np.sqrt(0.5))]
    err = np.abs(dev(3, s) / np.arcsin(s) - 1.0).max()
    assert err <= 2.0 ** -21, np.log2(err)

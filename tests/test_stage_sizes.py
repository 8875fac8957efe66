"""Shared memory of the sweep kernels: a block stages what its form reads and no more,
since every kilobyte is taken from L1.  The FP32 marches keep their cells in registers
and stage one cell and face ahead, whatever the reconstruction; the FP64 ones hold a
ring of four cells (PLM) or five (PPM)."""
import ctypes
import subprocess
import os

import pytest

from gpluto_dev_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))
MC, PPM, MP5 = 3, 4, 5


@pytest.fixture(scope="module")
def size(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("stage") / "stage_sizes.so")
    r = subprocess.run([build.nvcc(), *build.ARCH, *build.BASE, "-shared",
                        os.path.join(HERE, "stage_sizes.cu"), "-o", so], capture_output=True)
    assert r.returncode == 0, r.stderr.decode()[-2000:]
    lib = ctypes.CDLL(so)
    lib.stage_bytes.batch = lib.batch_bytes
    return lib.stage_bytes


@pytest.mark.parametrize("nv", [5, 8])
@pytest.mark.parametrize("lim", [MC, PPM, MP5])
def test_march(size, nv, lim):
    two = 2 * (nv + 1) * 128 * 8
    assert size(nv, lim, 1, 0) == two
    assert size(nv, lim, 0, 0) == {MC: (4 * nv + 2) * 128 * 8, PPM: (5 * nv + 2) * 128 * 8,
                                   MP5: two}[lim]


@pytest.mark.parametrize("nv", [5, 8])
def test_whole_fp32_rows(size, nv):
    assert size(nv, MC, 1, 2) == 2 * (2 * nv + 1) * 128 * 8
    assert size(nv, MC, 1, 2) < size(nv, MC, 1, 1) == size(nv, MC, 0, 1)


def test_batch_tiles_fit(size):
    """The batch's sweep launch stages the largest of its tiles, FP64 and FP32."""
    assert size.batch() == max(size(nv, MC, f, w) for nv in (5, 8) for f in (0, 1) for w in (0, 1, 2))

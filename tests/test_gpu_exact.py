"""FastArith (gp_exact.cuh) against the language's correctly rounded operators,
bit for bit: random significands over the exponent range it accepts, and the
arguments where it could go wrong -- all-ones and near-one significands,
quotients next to a rounding boundary, squares and their neighbours, zeros,
denormals, infinities and NaN (which have to set the flag)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
DIV, INV, ROOT, QUOT_POS, FIXED, DIV_ANY, SEEDS = range(7)


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("exact") / "exact_probe.so")
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-std=c++17", "-O3", "-fmad=false", "-shared", "-Xcompiler", "-fPIC",
                    os.path.join(HERE, "exact_probe.cu"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    lib.exact_probe.argtypes = [ctypes.c_void_p] * 5 + [ctypes.c_int] * 2

    def run(a, b, op):
        a = torch.as_tensor(a, dtype=torch.float64, device="cuda").contiguous()
        b = torch.as_tensor(b, dtype=torch.float64, device="cuda").contiguous()
        out, ref = torch.empty_like(a), torch.empty_like(a)
        bad = torch.empty(a.numel(), dtype=torch.int32, device="cuda")
        assert lib.exact_probe(a.data_ptr(), b.data_ptr(), out.data_ptr(), ref.data_ptr(),
                               bad.data_ptr(), a.numel(), op) == 0
        return out, ref, bad != 0
    return run


def _random(n, lo, hi, seed, near=False):
    g = torch.Generator(device="cuda").manual_seed(seed)
    m = torch.randint(0, 1 << 52, (n,), generator=g, device="cuda")
    if near:     # few bits set, or all but few: the neighbourhoods of powers of two
        m = torch.randint(0, 64, (n,), generator=g, device="cuda") \
            << torch.randint(0, 47, (n,), generator=g, device="cuda")
        flip = torch.randint(0, 2, (n,), generator=g, device="cuda")
        m = torch.where(flip == 1, ((1 << 52) - 1) - m, m) & ((1 << 52) - 1)
    e = torch.randint(lo, hi, (n,), generator=g, device="cuda")
    return (((e + 1023) << 52) | m).view(torch.float64)


def _same(out, ref, bad, most_bad):
    ok = ~bad
    assert torch.equal(out[ok].view(torch.int64), ref[ok].view(torch.int64))
    assert bad.double().mean().item() <= most_bad


@pytest.mark.parametrize("near", [False, True])
def test_random_arguments(probe, near):
    n = 1 << 24
    for seed in range(4):
        a, b = _random(n, -700, 700, seed, near), _random(n, -200, 200, 100 + seed, near)
        sign = torch.where(_random(n, 0, 2, 200 + seed) < 2, 1.0, -1.0).double()
        _same(*probe(a * sign, b, DIV), 0.0)
        _same(*probe(a, -b, DIV), 0.0)
        _same(*probe(a * sign, b, DIV_ANY), 0.0)
        _same(*probe(a, -b, DIV_ANY), 0.0)
        _same(*probe(a, b, INV), 0.0)
        _same(*probe(a, b, QUOT_POS), 0.0)
        _same(*probe(_random(n, -400, 400, 300 + seed, near), b, ROOT), 0.0)
        out, ref, _ = probe(a * sign, b, FIXED)
        assert torch.equal(out.view(torch.int64), ref.view(torch.int64))


def test_next_to_rounding_boundaries(probe):
    n = 1 << 22
    b = _random(n, 0, 1, 1)
    q = _random(n, 0, 1, 2)
    for k in (-2, -1, 0, 1, 2):   # dividends whose quotient is q to within an ulp or so
        a = ((q * b).view(torch.int64) + k).view(torch.float64)
        _same(*probe(a, b, DIV), 0.0)
        _same(*probe(-a, b, DIV_ANY), 0.0)
        s = ((q * q).view(torch.int64) + k).view(torch.float64)   # roots next to q
        _same(*probe(s, b, ROOT), 0.0)


def test_special_values(probe):
    tiny, inf, nan = 5e-324, float("inf"), float("nan")
    for a, b in ((0.0, 3.0), (-0.0, 3.0), (0.0, -3.0), (-0.0, -3.0)):
        for op in (DIV, DIV_ANY):
            out, ref, bad = probe([a], [b], op)
            assert not bad.any() and torch.equal(out.view(torch.int64), ref.view(torch.int64))
    ones = np.nextafter(2.0, 0.0)
    for a in (1.0, ones, np.nextafter(ones, 0.0), 3.0, -ones):
        for b in (ones, ones / 2, -ones, np.nextafter(ones, 0.0)):
            for op in (DIV, INV):
                out, ref, bad = probe([a], [b], op)
                assert not bad.any() and torch.equal(out.view(torch.int64),
                                                     ref.view(torch.int64))
    for a, b in ((1.0, 0.0), (1.0, tiny), (1.0, inf), (1.0, nan), (tiny, 1.0),
                 (1e-320, 3.0), (inf, 1.0), (nan, 1.0), (1e-250, 1.0), (1e250, 1.0),
                 (1.0, 1e70), (1.0, 1e-70)):
        assert probe([a], [b], DIV)[2].all() and probe([a], [b], DIV_ANY)[2].all()
        out, ref, bad = probe([a], [b], FIXED)    # falls back by itself
        assert torch.equal(out.view(torch.int64), ref.view(torch.int64)) or np.isnan(a + b)
    for a in (0.0, -0.0, -1.0, tiny, 1e-320, inf, nan, 1e-130, 1e130):
        assert probe([a], [1.0], ROOT)[2].all()
        assert a > 0 or probe([a], [1.0], QUOT_POS)[2].all()


def test_seed_errors(probe):
    """The seeds are as good as gp_exact.cuh's derivation needs: e = 1 - b y0 with
    |e|^3 <= 2^-58, and e = 1 - a y0^2 with 5/16 |e|^3 <= 2^-57.4 (0.05 ulp of a root's
    iterate).  They are functions of an argument's upper 20 significand bits: all of
    those, the rest zero or ones, both parities of the exponent."""
    top = torch.arange(1 << 20, device="cuda", dtype=torch.int64) << 32
    m = torch.cat([top, top | 0xffffffff])
    a = torch.cat([m | (1023 << 52), m | (1024 << 52)]).view(torch.float64)
    rcp, rsqrt, _ = probe(a, a, SEEDS)
    assert rcp.abs().max().item() ** 3 <= 2.0 ** -58
    assert 5.0 / 16.0 * rsqrt.abs().max().item() ** 3 <= 2.0 ** -57.4

"""csrc/exact_div.cuh against CUDA's own exactly rounded reciprocal and quotient:
every bit (the sign of zeros included), over random operands of the whole range,
significands of all ones and their neighbours, operands on both sides of the
limits of the shared-reciprocal path, zeros, subnormals, infinities and NaN."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ONES = (1 << 52) - 1


@pytest.fixture(scope="module")
def lib(gpu, tmp_path_factory):
    out = tmp_path_factory.mktemp("exact_div") / "libexact_div_check.so"
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "-fmad=false", "-shared", "-Xcompiler", "-fPIC",
                    "-I" + os.path.join(ROOT, "verb-4d_b200", "csrc"),
                    os.path.join(ROOT, "tests", "exact_div_check.cu"), "-o", str(out)], check=True)
    return ctypes.CDLL(str(out))


def value(exponent, significand, negative=None):
    """2^exponent (1 + significand / 2^52)"""
    bits = ((np.asarray(exponent, np.int64) + 1023) << 52) | np.asarray(significand, np.int64)
    v = bits.view(np.float64)
    return v if negative is None else np.where(negative, -v, v)


def run(lib, a, b):
    import torch

    a, b = np.broadcast_arrays(a, b)
    d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (a, b)]
    out = [torch.empty_like(d[0]) for _ in range(4)]
    torch.cuda.synchronize()
    p = [ctypes.c_void_p(t.data_ptr()) for t in d + out]
    assert lib.exact_div_check(p[0], p[1], ctypes.c_size_t(a.size), *p[2:]) == 0
    return [t.cpu().numpy() for t in out]


def same(x, y):
    return (x.view(np.int64) == y.view(np.int64)) | (np.isnan(x) & np.isnan(y))


def significands(rng, n):
    s = rng.integers(0, 1 << 52, n)
    few = rng.integers(0, 256, n) << rng.integers(0, 45, n)   # few bits: exact and halfway quotients
    near = np.where(rng.random(n) < 0.5, ONES - rng.integers(0, 3, n), rng.integers(0, 3, n))
    kind = rng.integers(0, 3, n)
    return np.where(kind == 0, s, np.where(kind == 1, few & ONES, near))


def test_random_operands(lib):
    rng = np.random.default_rng(1)
    n = 1 << 22
    for span in (4, 405, 1021):  # inside the limits, across them, everything
        a = value(rng.integers(-span, span + 1, n), significands(rng, n), rng.random(n) < 0.5)
        b = value(rng.integers(-span, span + 1, n), significands(rng, n), rng.random(n) < 0.5)
        q, ref, y, yref = run(lib, a, b)
        assert same(q, ref).all(), (a[~same(q, ref)][:3], b[~same(q, ref)][:3])
        assert same(y, yref).all(), b[~same(y, yref)][:3]


def test_significands_of_all_ones(lib):
    e = np.arange(-1021, 1022)
    b = np.concatenate([value(e, np.full(e.size, ONES - k)) for k in range(3)])
    _, _, y, yref = run(lib, np.ones(b.size), b)
    assert same(y, yref).all(), b[~same(y, yref)][:3]


def test_edges(lib):
    edge = []
    for e in (-1022, -401, -400, -399, -1, 0, 1, 399, 400, 401, 1023):
        for s in (0, 1, ONES - 1, ONES):
            edge.append(float(value(e, s)))
    edge += [0.0, 5e-324, 2.2e-308, np.inf, np.nan]
    edge = np.array(edge + [-x for x in edge])
    a, b = (g.ravel() for g in np.meshgrid(edge, edge))
    q, ref, _, _ = run(lib, a, b)
    assert same(q, ref).all(), (a[~same(q, ref)][:5], b[~same(q, ref)][:5])

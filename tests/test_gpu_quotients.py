"""The branch-free quotients and roots of cb_div.cuh against IEEE division and
square root, bit for bit, and the mixed form's packed reconstructions against
their scalar functions.

FP64.  For denominators and radicands in 2^-960 .. 2^960 the corrected quotient
q + (a - b q) y has the IEEE bits unless a / b lies within d of a rounding
boundary.  The remainder is exact and below 2^0.6 ulp of q times b, and y is
1 / b to a relative 2^-52.9 (its cubic step leaves 2^-59, its rounding 2^-53),
so d < 2^-52 ulp.  For the root the remainder x - g^2 is itself rounded
(relative 2^-53) and h is 1 / (2 g) to 2^-51.4 (two roundings behind a cubic
step), so d < 2^-50 ulp.  Random operands come that near a boundary once in
2^50; operands built from a boundary do, and may be off by one ulp there."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
QUOT, ROOT, THIRD, BY27 = range(4)


def _build(tmp, flags, name):
    from chimera_comp_les_b200 import build as B
    so = str(tmp / (name + ".so"))
    cmd = [B.NVCC, *B.NVCC_FLAGS, *flags, "-shared", "-I", os.path.join(B.PKG_DIR, "csrc"), "-o", so,
           os.path.join(HERE, "cuda", "quotient_probe.cu")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(so)


@pytest.fixture(scope="module")
def fp64(tmp_path_factory):
    from chimera_comp_les_b200 import build as B
    lib = _build(tmp_path_factory.mktemp("probe64"), B.FP64_FLAGS, "probe64")

    def call(op, a, b=None):
        a = np.ascontiguousarray(a, np.float64)
        b = np.ones_like(a) if b is None else np.ascontiguousarray(b, np.float64)
        out = np.full_like(a, np.nan)
        p = ctypes.POINTER(ctypes.c_double)
        assert lib.probe_fp64(op, a.ctypes.data_as(p), b.ctypes.data_as(p), out.ctypes.data_as(p), a.size) == 0
        return out
    return call


@pytest.fixture(scope="module")
def mixed(tmp_path_factory):
    from chimera_comp_les_b200 import build as B
    return _build(tmp_path_factory.mktemp("probe32"), B.MIXED_FLAGS, "probe32")


def _random(rng, n, lo, hi):
    """Signed values of exponents lo .. hi - 1, a part of them with mantissas at the ends of a binade."""
    m = rng.random(n) + 1.0
    edge = rng.integers(0, 8, n) == 0
    m[edge] = rng.choice([1.0, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52, 1.5], int(edge.sum()))
    return np.ldexp(m, rng.integers(lo, hi, n)) * rng.choice([-1.0, 1.0], n)


def _ulps(got, want):
    return np.abs(got.view(np.int64) - want.view(np.int64))


@pytest.mark.parametrize("span", [3, 400, 960])
def test_random_quotients_have_the_ieee_bits(fp64, span):
    rng = np.random.default_rng(span)
    n = 1 << 22
    b = _random(rng, n, -span, span)
    a = _random(rng, n, -60, 60) if span == 960 else _random(rng, n, -span, span)
    off = _ulps(fp64(QUOT, a, b), a / b)
    # a power of two over a mantissa of ones, 2^-54 ulp beside a boundary
    near = (np.abs(np.frexp(a)[0]) == 0.5) & (np.abs(np.frexp(b)[0]) == 1.0 - 2.0 ** -53)
    assert off[near].max() <= 1
    assert not off[~near].any()


@pytest.mark.parametrize("span", [2, 960])
def test_random_roots_have_the_ieee_bits(fp64, span):
    x = np.abs(_random(np.random.default_rng(span), 1 << 22, -span, span))
    assert np.array_equal(fp64(ROOT, x).view(np.int64), np.sqrt(x).view(np.int64))


@pytest.mark.parametrize("op,den", [(THIRD, 3.0), (BY27, 27.0)])
def test_quotients_by_constants_have_the_ieee_bits(fp64, op, den):
    a = _random(np.random.default_rng(op), 1 << 22, -900, 900)
    assert np.array_equal(fp64(op, a).view(np.int64), (a / den).view(np.int64))


def test_quotients_next_to_a_rounding_boundary(fp64):
    """a / b = (m - c / b) 2^-54 with m odd: the boundary m, missed by c / b of half an ulp."""
    rng = np.random.default_rng(7)
    A, B, C = [], [], []
    while len(A) < 40000:
        b = int(rng.integers(1 << 52, 1 << 53)) | 1
        c = int(rng.integers(1, 200)) * int(rng.choice([-1, 1]))
        m = c * pow(b, -1, 1 << 54) % (1 << 54)  # m b = c mod 2^54
        if m % 2 == 0 or m < 1 << 53:
            continue
        a = (m * b - c) >> 54
        if a >= 1 << 53:
            continue
        A.append(float(a)); B.append(float(b)); C.append(c)
    a, b, c = np.array(A), np.array(B), np.abs(np.array(C))
    off = _ulps(fp64(QUOT, a, b), a / b)
    assert off.max() <= 1
    assert not off[0.5 * c / b > 2.0 ** -52].any()


def test_roots_next_to_a_rounding_boundary(fp64):
    """x = (M^2 + c) with M odd of 54 bits and x of 53: sqrt(x) = M + c / (2 M), the boundary M missed by c / (2 M) of
    half an ulp."""
    X, D = [], []
    for c in range(7, 40000, 8):  # -c = 1 mod 8: M^2 = -c has odd solutions mod every power of two
        r = 1
        for k in range(3, 57):  # r^2 = -c mod 2^k -> mod 2^(k + 1)
            if (r * r + c) % (1 << (k + 1)):
                r += 1 << (k - 1)
        for m in (r, (1 << 57) - r, r + (1 << 56), (1 << 57) - r + (1 << 56)):
            m %= 1 << 57
            if not 1 << 53 <= m < 1 << 54:
                continue
            x = m * m + c
            if x % (1 << (x.bit_length() - 53)) == 0:
                X.append(float(x)); D.append(0.5 * c / (2 * m))
    x, d = np.array(X), np.array(D)
    assert x.size > 500
    off = _ulps(fp64(ROOT, x), np.sqrt(x))
    assert off.max() <= 1
    assert not off[d > 2.0 ** -50].any()


def _stencils(rng, n, kind):
    if kind == "smooth":
        t = rng.random((n, 2, 1)) * 6.28 + np.arange(6) * 0.2
        return (1.0 + 0.3 * np.sin(t)).astype(np.float32)
    if kind == "plateaus":
        return (0.25 * rng.integers(-2, 3, (n, 2, 6))).astype(np.float32)
    v = rng.standard_normal((n, 2, 6)) * 10.0 ** rng.uniform(-6, 6, (n, 2, 1))
    return v.astype(np.float32)


@pytest.mark.parametrize("kind", ["smooth", "plateaus", "rough"])
@pytest.mark.parametrize("op", [0, 1, 2], ids=["muscl", "weno3", "weno5"])
def test_packed_reconstructions_have_the_scalar_bits(mixed, op, kind):
    n = 1 << 20
    v = np.ascontiguousarray(_stencils(np.random.default_rng(op), n, kind))
    out = np.empty((n, 8), np.float32)
    p = ctypes.POINTER(ctypes.c_float)
    assert mixed.probe_recon(op, v.ctypes.data_as(p), out.ctypes.data_as(p), n) == 0
    assert np.isfinite(out).all()
    assert np.array_equal(out[:, :4].view(np.int32), out[:, 4:].view(np.int32))


def test_fp32_quotients_have_the_fast_division_bits(mixed):
    """Denominators of exponents -120 .. 119, quotients in range; 1 / b and the root alike."""
    rng = np.random.default_rng(1)
    n = 1 << 22
    b = np.ldexp(1.0 + rng.random(n), rng.integers(-120, 120, n)).astype(np.float32)
    a = (np.ldexp(1.0 + rng.random(n), rng.integers(-3, 4, n)) * rng.choice([-1, 1], n)).astype(np.float32)
    out = np.empty((n, 6), np.float32)
    p = ctypes.POINTER(ctypes.c_float)
    assert mixed.probe_fp32(a.ctypes.data_as(p), b.ctypes.data_as(p), out.ctypes.data_as(p), n) == 0
    for x in (0, 2, 4):
        assert np.array_equal(out[:, x].view(np.int32), out[:, x + 1].view(np.int32))

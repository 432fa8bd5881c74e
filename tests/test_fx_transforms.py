"""Fixed-point transforms of the FP64 form (ps3d_gb300/csrc/fx.cuh) against
dense transform matrices in extended precision: the host build of the device
functions on the CPU, the kernels on the GPU.

Tolerance: the conversion of each output rounds once (2^-53 of its size), and
at most four passes round by one unit, which on the lines used here is at
most 2^-54 of the rms output: (2^-53 + 4 * 2^-54) relative L2.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "ps3d_gb300", "csrc")
TOL = 2.0 ** -53 + 4 * 2.0 ** -54
LD = np.longdouble
PI = np.arccos(LD(-1))


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    lib = str(tmp_path_factory.mktemp("fx") / "libfx.so")
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-std=c++17", "-I/usr/local/cuda/include", "-I", CSRC, "-o", lib,
                    os.path.join(HERE, "fx_host.cpp")], check=True)
    L = ctypes.CDLL(lib)

    def call(fn, n, flag, wide, a, b):
        out = [np.zeros_like(a), np.zeros_like(b)]
        p = [x.ctypes.data_as(ctypes.c_void_p) for x in (a, b, *out)]
        getattr(L, fn)(n, flag, wide, *p)
        return out

    return call


def rel(x, ref):
    return float(np.sqrt(np.sum((x.astype(LD) - ref) ** 2) / np.sum(ref ** 2)))


def fourier(n):
    """forward and inverse in the Hermitian storage (cosine rows 0..n/2, then
    the sine parts mirrored), scale 1/sqrt(n) both ways"""
    k = np.arange(n)
    a = (np.outer(np.minimum(k, n - k), k) % n).astype(LD) * (2 * PI / n)
    f = np.where((k <= n // 2)[:, None], np.cos(a), -np.sin(a)) / np.sqrt(LD(n))
    w = np.full(n, LD(2))
    w[0] = w[n // 2] = 1
    return f, (f * w[:, None]).T


def sine_cosine(n):
    j = np.arange(n + 1)
    a = (np.outer(j, j) % (2 * n)).astype(LD) * (PI / n)
    s, c = np.sin(a) * np.sqrt(LD(2) / n), np.cos(a) * np.sqrt(LD(2) / n)
    s[0] = s[n] = s[:, 0] = s[:, n] = 0
    c[:, 0] /= 2
    c[:, n] /= 2
    return s, c


def line(kind, n, rng):
    k = np.minimum(np.arange(n), n - np.arange(n))
    return {"noise": lambda: rng.standard_normal(n),
            "spectrum": lambda: rng.standard_normal(n) * np.exp(-0.5 * k),
            "spike": lambda: np.where(np.arange(n) == 3, 1.7, 1e-3 * rng.standard_normal(n)),
            "offset": lambda: 1e6 + rng.standard_normal(n)}[kind]()


KINDS = ["noise", "spectrum", "spike", "offset"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [8, 10, 12, 18, 30, 60, 96, 128, 250, 256, 288, 512])
def test_lines_host(host, n, kind):
    rng = np.random.default_rng(n)
    a, b = line(kind, n, rng), 1e-9 * line(kind, n, rng)
    for inverse, m in enumerate(fourier(n)):
        oa, ob = host("fx_line", n, inverse, inverse, a, b)
        assert rel(oa, m @ a.astype(LD)) < TOL and rel(ob, m @ b.astype(LD)) < TOL, inverse


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [8, 10, 12, 30, 60, 96, 128, 256, 288, 512])
def test_columns_host(host, n, kind):
    rng = np.random.default_rng(n)
    a, b = line(kind, n + 1, rng), 1e9 * line(kind, n + 1, rng)
    for dct, m in enumerate(sine_cosine(n)):
        oa, ob = host("fx_column", n, dct, 1 - dct, a, b)
        assert rel(oa, m @ a.astype(LD)) < TOL and rel(ob, m @ b.astype(LD)) < TOL, dct


@pytest.mark.parametrize("scale", [1e-305, 1e-290, 1e-150, 1e150, 1e300])
def test_scales_and_non_finite_lines(host, scale):
    """any magnitude, zero lines exactly, a non-finite value only in its own line"""
    n = 48
    rng = np.random.default_rng(7)
    f, _ = fourier(n)
    a = rng.standard_normal(n) * scale
    oa, ob = host("fx_line", n, 0, 1, a, np.zeros(n))
    tol = TOL if scale > 1e-300 else 1e-2 * 2.0 ** -1022 / scale  # subnormal outputs
    assert rel(oa / LD(scale), f @ (a / LD(scale))) < tol and not ob.any()
    for bad in (np.nan, np.inf, -np.inf):
        c = rng.standard_normal(n)
        c[5] = bad
        oc, oa2 = host("fx_line", n, 0, 1, c, a)
        assert np.isnan(oc).all() and rel(oa2 / LD(scale), f @ (a / LD(scale))) < tol


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(8, 10, 8), (12, 30, 10), (60, 8, 288), (32, 32, 30), (128, 12, 72), (8, 512, 12),
                                   (10, 24, 512), (18, 250, 24), (500, 54, 8)])
def test_operators_device(shape):
    """every tile tail: odd z counts, few pairs per block, ragged columns"""
    from ps3d_gb300 import Ps3dGpu
    nx, ny, nz = shape
    g = Ps3dGpu(nx, ny, nz, (0.0, 0.0, 0.0), (2.0, 3.0, 1.0))
    rng = np.random.default_rng(nx + ny)
    f = rng.standard_normal((nx, ny, nz + 1)) * np.exp(rng.uniform(-20, 20, (1, 1, nz + 1)))
    ld = f.astype(LD)
    (fx, ix), (fy, iy) = fourier(nx), fourier(ny)
    for op, mx, my in (("fftxyp2s", fx, fy), ("fftxys2p", ix, iy)):
        out = getattr(g, op)(f)
        ref = np.einsum("ai,bj,ijk->abk", mx, my, ld, optimize=True)
        for k in range(nz + 1):  # every level by its own size: two passes
            assert rel(out[..., k], ref[..., k]) < 2 * TOL, (op, k)
    s, c = sine_cosine(nz)
    out = g.fftsine(f)
    assert rel(out[..., 1:nz], (ld @ s.T)[..., 1:nz]) < TOL
    assert np.array_equal(out[..., 0], f[..., 0]) and not out[..., nz].any()
    assert rel(g.fftcosine(f), ld @ c.T) < TOL
    f[1, 1, 2] = np.nan
    out = g.fftxyp2s(f)
    assert np.isnan(out[..., 2]).all() and np.isfinite(np.delete(out, 2, axis=2)).all()
    g.close()

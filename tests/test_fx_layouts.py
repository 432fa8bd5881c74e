"""Fixed-point transforms in the layouts that test_fx_transforms.py leaves
out: eight pairs of lines per block, in two buffers (below 128 points) and in
one, with ragged levels; non-finite values in columns.  Tolerances as there."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from tests.test_fx_transforms import CSRC, HERE, KINDS, LD, TOL, fourier, line, rel, sine_cosine


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    lib = str(tmp_path_factory.mktemp("fxw") / "libfxw.so")
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-std=c++17", "-I/usr/local/cuda/include", "-I", CSRC, "-I", HERE,
                    "-o", lib, os.path.join(HERE, "fx_host_wide.cpp")], check=True)
    L = ctypes.CDLL(lib)

    def call(fn, n, flag, wide, a, b):
        out = [np.zeros_like(a), np.zeros_like(b)]
        getattr(L, fn)(n, flag, wide, *(x.ctypes.data_as(ctypes.c_void_p) for x in (a, b, *out)))
        return out

    return call


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [36, 80, 96, 100, 128, 144, 160, 240, 256])
def test_eight_pairs_host(host, n, kind):
    rng = np.random.default_rng(n)
    a, b = line(kind, n, rng), 1e-9 * line(kind, n, rng)
    for inverse, m in enumerate(fourier(n)):
        oa, ob = host("fx_line_wide", n, inverse, 0, a, b)
        assert rel(oa, m @ a.astype(LD)) < TOL and rel(ob, m @ b.astype(LD)) < TOL, inverse


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("n", [12, 64, 270])
def test_non_finite_column_host(host, n, bad):
    """a non-finite value makes its own column NaN and leaves the one packed with it"""
    rng = np.random.default_rng(n)
    a, b = rng.standard_normal(n + 1), rng.standard_normal(n + 1)
    a[n // 3] = bad
    for dct, m in enumerate(sine_cosine(n)):
        for pair, own in (((a, b), 0), ((b, a), 1)):
            out = host("fx_column", n, dct, 1 - dct, *pair)
            assert np.isnan(out[own][1:n]).all() and rel(out[1 - own], m @ b.astype(LD)) < TOL, dct


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(96, 144, 60), (144, 80, 60), (100, 80, 60)])
def test_eight_pairs_device(shape):
    """grids at which the rule of fx_lines takes eight pairs on both axes"""
    from ps3d_gb300 import Ps3dGpu
    nx, ny, nz = shape
    g = Ps3dGpu(nx, ny, nz, (0.0, 0.0, 0.0), (2.0, 3.0, 1.0))
    rng = np.random.default_rng(nx)
    f = rng.standard_normal((nx, ny, nz + 1)) * np.exp(rng.uniform(-20, 20, (1, 1, nz + 1)))
    levels = [0, 1, 15, 16, nz - 1, nz]  # first, tile edges, last
    ld = f[..., levels].astype(LD)
    (fx, ix), (fy, iy) = fourier(nx), fourier(ny)
    for op, mx, my in (("fftxyp2s", fx, fy), ("fftxys2p", ix, iy)):
        out = getattr(g, op)(f)
        ref = np.einsum("ai,bj,ijk->abk", mx, my, ld, optimize=True)
        for q, k in enumerate(levels):  # every level by its own size: two passes
            assert rel(out[..., k], ref[..., q]) < 2 * TOL, (op, k)
    g.close()


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(8, 10, 32), (96, 72, 96), (8, 8, 270)])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_column_device(shape, bad):
    from ps3d_gb300 import Ps3dGpu
    nx, ny, nz = shape
    g = Ps3dGpu(nx, ny, nz, (0.0, 0.0, 0.0), (2.0, 3.0, 1.0))
    f = np.random.default_rng(nz).standard_normal((nx, ny, nz + 1))
    for op in ("fftsine", "fftcosine", "decompose_semi_spectral", "combine_semi_spectral"):
        clean = getattr(g, op)(f)
        h = f.copy()
        h[1, 3, nz // 3] = bad
        out = getattr(g, op)(h)
        assert np.isnan(out[1, 3, 1:nz]).all(), op
        # (1, 2) is packed with it and shares its roundings
        assert rel(out[1, 2], clean[1, 2].astype(LD)) < 2 * TOL, op
        out[1, 2:4], clean[1, 2:4] = 0.0, 0.0
        assert np.array_equal(out, clean), op
    g.close()

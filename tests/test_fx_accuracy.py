"""The fixed-point transforms (ps3d_gb300/csrc/fx.cuh) are no less accurate
than the FP64 Stockham transforms in whose place they run: on the spectra the
solver meets, at lengths with many small factors and up to the longest they
serve, the root mean square over 40 lines of the relative error against dense
transforms in extended precision is at most the FP64 transforms' on the same
lines.  Lines that reach the bounds of the plan do not overflow."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from tests.test_fx_transforms import CSRC, HERE, LD, fourier, rel, sine_cosine

KINDS = {"noise": 0.0, "k^-5/6": -5 / 6, "k^-5/3": -5 / 3, "k^-2": -2.0, "k^-4": -4.0}
LENGTHS = [64, 96, 128, 250, 256, 270, 324, 360, 400, 432, 450, 480, 486, 500, 512]


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    libs = {}
    for name in ("fx", "fp64"):
        lib = str(tmp_path_factory.mktemp("host") / ("lib%s.so" % name))
        subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-std=c++17", "-ffp-contract=off",
                        "-I/usr/local/cuda/include", "-I", CSRC, "-o", lib,
                        os.path.join(HERE, name + "_host.cpp")], check=True)
        libs[name] = ctypes.CDLL(lib)

    def call(form, what, n, flag, a, b):
        out = [np.zeros_like(a), np.zeros_like(b)]
        p = [x.ctypes.data_as(ctypes.c_void_p) for x in (a, b, *out)]
        getattr(libs[form], "%s_%s" % (form, what))(n, flag, int(n <= 128), *p)
        return out

    return call


def draw(rng, k, power):
    return rng.standard_normal(k.size) * np.maximum(k, 1.0) ** power


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", LENGTHS)
def test_error_is_at_most_the_fp64_transforms(host, n, kind):
    rng = np.random.default_rng(n)
    j = np.arange(n)
    for what, mats, k in (("line", fourier(n), np.minimum(j, n - j)), ("column", sine_cosine(n), np.arange(n + 1))):
        for flag, m in enumerate(mats):
            err = {"fx": [], "fp64": []}
            for _ in range(20):
                pair = [draw(rng, k, KINDS[kind]) for _ in range(2)]
                refs = [m @ x.astype(LD) for x in pair]
                for form in err:
                    outs = host(form, what, n, flag, *pair)
                    err[form] += [rel(o, r) if flag or what == "line" else rel(o[1:n], r[1:n])
                                  for o, r in zip(outs, refs)]
            fx, fp64 = (float(np.sqrt(np.mean(np.square(err[f])))) for f in ("fx", "fp64"))
            assert fx <= fp64, (what, flag, fx, fp64)


@pytest.mark.parametrize("n", [8, 10, 12, 18, 30, 48, 54, 96, 128, 160, 250, 256, 288, 324, 400, 432, 486, 500, 512])
def test_no_overflow_at_the_bounds(host, n):
    """values of the largest significand, signed so that one output adds them
    all up: every value, and so few that their sum just stays below a power of
    two; a constant line, alternating signs and single values"""
    top = np.nextafter(2.0, 0.0)
    for what, mats, size in (("line", fourier(n), n), ("column", sine_cosine(n), n + 1)):
        for flag, m in enumerate(mats):
            rows = m.astype(np.float64)
            lo, hi = (1, n) if what == "column" and not flag else (0, size)
            lines = [np.full(size, top), top * (-1.0) ** np.arange(size)]
            for k in sorted({lo, lo + 1, lo + 2, n // 8, n // 4, n // 3, n // 2, n - 2, hi - 1}):
                sign = np.where(rows[k] < 0, -top, top)
                order = np.argsort(-np.abs(rows[k]), kind="stable")
                for count in (1, 2, 3, 4, 8, 15, 16, 31, 32, 64, 127, 128, 255, 256, size):
                    x = np.zeros(size)
                    x[order[:count]] = sign[order[:count]]
                    lines.append(x)
            for i, a in enumerate(lines):
                b = lines[-1 - i]
                for x, y in ((a, a), (a, -a), (a, b)):
                    outs = host("fx", what, n, flag, x.copy(), y.copy())
                    for o, z in zip(outs, (x, y)):
                        r = m @ z.astype(LD)
                        norm = np.sqrt(np.sum(z.astype(LD) ** 2))
                        assert np.sqrt(np.sum((o[lo:hi] - r[lo:hi]) ** 2)) <= 1e-15 * norm, (what, flag, i)

"""The register fronts' barriers, on the CPU: tests/register_front_host.cpp
runs the CTA's threads under schedules in which some warps run as far ahead as
the barriers let them, and compares every result with the same factorization
written as plain loops. Consecutive candidates that do not pass where they
stand (interchanges, 2x2 pivots, delays) are what the schedules are for: a
warp that meets the second of them early must not touch what the others still
read for the first. The arithmetic is the same operation for operation, so
the entries have to be equal."""

import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "amigo_b200", "csrc")


def _cuda_include():
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    return os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None or not os.path.exists(os.path.join(_cuda_include(), "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    so = str(tmp_path_factory.mktemp("front") / "front.so")
    subprocess.run([cxx, "-std=c++17", "-O1", "-mfma", "-ffp-contract=off", "-w", "-fPIC",
                    "-shared", "-I", _cuda_include(), "-I", CSRC,
                    os.path.join(HERE, "register_front_host.cpp"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    lib.front_schedules.argtypes = [ctypes.c_int] * 5 + [ctypes.c_double] * 2 + [
        ctypes.POINTER(ctypes.c_double), ctypes.c_uint, ctypes.c_uint,
        ctypes.POINTER(ctypes.c_int), ctypes.c_char_p, ctypes.c_int]
    return lib


def _matrix(kind, f, fs, seed):
    rng = np.random.default_rng(seed)
    a = rng.standard_normal((f, f))
    a = a + a.T
    d = np.arange(f)
    if kind == "zeros":  # a third of the diagonal
        a[d[::3], d[::3]] = 0.0
    elif kind == "small":  # hardly any candidate passes where it stands
        a[d, d] *= 1e-3
    elif kind == "block":  # half of the candidates far below the rows they meet
        a[:fs // 2, :fs // 2] *= 1e-9
    elif kind == "definite":
        a = a @ a.T + f * np.eye(f)
    return np.asfortranarray(a)


def _check(lib, a, fs, root, cholesky, ustab, schedules):
    f = a.shape[0]
    chunks = 1 if f <= 32 else 2 if f <= 64 else 3 if f <= 96 else 5
    out = (ctypes.c_int * 5)()
    why = ctypes.create_string_buffer(80)
    bad = lib.front_schedules(chunks, f, fs, root, cholesky, ustab, 1e-14,
                              a.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), 0, schedules,
                              out, why, len(why))
    assert bad == 0, f"schedule {bad - 1}: {why.value.decode()}"
    return dict(zip(("pivots", "pos", "neg", "pairs", "moved"), out))


@pytest.mark.parametrize("kind", ["zeros", "small"])
@pytest.mark.parametrize("f", [1, 2, 7, 8, 9, 32, 33, 64, 65, 96, 97, 128, 143, 144])
def test_root(lib, f, kind):
    """Bunch-Kaufman: 1x1 pivots at imax and 2x2 pivots one after another."""
    out = _check(lib, _matrix(kind, f, f, f), f, 1, 0, 0.01, 8)
    assert out["pivots"] == f
    if f >= 32 and kind == "small":
        assert out["pairs"] > 5 and out["moved"] > 10


@pytest.mark.parametrize("ustab", [0.01, 0.4])
@pytest.mark.parametrize("kind", ["small", "block"])
@pytest.mark.parametrize("f,fs", [(9, 8), (20, 12), (33, 33), (40, 30), (64, 1), (70, 60),
                                  (97, 64), (144, 100)])
def test_candidates_and_rows(lib, f, fs, kind, ustab):
    """Threshold pivoting: interchanges, 2x2 pivots and delays."""
    _check(lib, _matrix(kind, f, fs, 100 * f + fs), fs, 0, 0, ustab, 8)


@pytest.mark.parametrize("f,fs", [(8, 8), (33, 20), (96, 96), (130, 70)])
def test_cholesky(lib, f, fs):
    out = _check(lib, _matrix("definite", f, fs, f), fs, 0, 1, 0.01, 6)
    assert out["pivots"] == out["pos"] == fs and out["moved"] == 0


@pytest.mark.parametrize("root", [0, 1])
@pytest.mark.parametrize("f,at", [(6, 2), (40, 0), (40, 39), (70, 33)])
@pytest.mark.parametrize("what", ["isolated nan", "nan", "isolated inf", "inf", "nan row",
                                  "isolated zero", "tiny"])
def test_values_that_are_not_numbers(lib, f, at, what, root):
    """Not-a-number, infinite and zero entries take the pivots that the plain
    loops take (a pivot column that is zero or not a number throughout counts
    as a zero pivot at a root, and leaves the other rows as they are)."""
    a = _matrix("zeros", f, f, f + at)
    if what.startswith("isolated"):
        a[at, :] = a[:, at] = 0.0
    value = {"nan": np.nan, "inf": np.inf, "zero": 0.0, "tiny": 1e-310}
    if what == "nan row":
        a[at, :] = a[:, at] = np.nan
    else:
        a[at, at] = value[what.split()[-1]]
    if what == "inf":
        a[(at + 1) % f, at] = a[at, (at + 1) % f] = -np.inf
    _check(lib, a, f if root else f - 2, root, 0, 0.01, 2)

"""The FP64 factorisation's reciprocal and root against CUDA's, over all
positive finite numbers: random mantissas at every exponent, subnormals, powers
of two and their neighbours, values next to 1 and 4.  The reciprocal's last
operation adds a correction below 2^-20 of it to the approximation, so it is
within one unit in the last place (half of it that operation's rounding, and
2^-60 of it the series) of the quotient, itself rounded; the same holds for the
root, and for the inverse root as the quotient 1 / root."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CSRC = os.path.join(ROOT, "3dreconstruction_gb300", "csrc")
SRC = os.path.join(ROOT, "tests", "device", "pivot_check.cu")


def pivots():
    rng = np.random.default_rng(7)
    e = np.repeat(np.arange(1, 2047, dtype=np.uint64), 200)
    random = (e << np.uint64(52)) | rng.integers(0, 1 << 52, e.size, dtype=np.uint64)
    subnormal = rng.integers(1, 1 << 52, 20000, dtype=np.uint64) >> rng.integers(0, 52, 20000, dtype=np.uint64)
    power = np.concatenate([np.arange(1, 2047, dtype=np.uint64) << np.uint64(52),
                            np.uint64(1) << np.arange(52, dtype=np.uint64)])
    near = np.concatenate([np.array([v], np.float64).view(np.uint64) + np.arange(-2000, 2001).astype(np.uint64)
                           for v in (1.0, 2.0, 4.0, 2.0**-900, 2.0**900)])
    bits = np.concatenate([random, subnormal, power, power - np.uint64(1), power + np.uint64(1), near])
    d = np.unique(bits).view(np.float64)
    return d[(d > 0) & np.isfinite(d)]


def test_reciprocal_and_root_within_a_unit(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "check")
    subprocess.run([nvcc, "-gencode=arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-I", CSRC, SRC, "-o", exe],
                   check=True, capture_output=True)
    d = pivots()
    d.tofile(tmp_path / "in")
    subprocess.run([exe, str(tmp_path / "in"), str(tmp_path / "out")], check=True, timeout=120)
    rcp, root, inv, q, s = np.fromfile(tmp_path / "out", np.float64).reshape(5, -1)
    with np.errstate(over="ignore"):
        np.testing.assert_array_equal(q, 1.0 / d)
        np.testing.assert_array_equal(s, np.sqrt(d))
    fin = np.isfinite(q)
    assert np.isinf(rcp[~fin]).all()
    assert (np.abs(rcp[fin] - q[fin]) <= np.spacing(q[fin])).all()
    assert (np.abs(root - s) <= np.spacing(s)).all()
    assert (np.abs(inv - 1.0 / root) <= np.spacing(inv)).all()

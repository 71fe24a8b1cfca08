"""The FP64 estimators' short form (Householder blocks, moments, inverse
iteration, FP32 sweeps for the sign) against the general form, on the CPU:
where the short form takes a track its vector has the general form's sign and
is within 1e-11 of it (both are accurate to about 1e-16 times the ratio of the
design's largest singular value to the gap, below 1e5 for these tracks), and
it takes nearly all tracks of ordinary noise.  Tracks that it must leave alone
(one view, no view, a view repeated, residuals as large as the depths) come
back untaken or equal."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "3dreconstruction_gb300", "csrc")
SRC = os.path.join(ROOT, "tests", "host", "tri_short_check.cu")


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    e = str(tmp_path_factory.mktemp("tri") / "check")
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-O2", "-x", "cu", "-I", CSRC, SRC, "-o", e],
                   check=True, capture_output=True)
    return e


def run(exe, tmp_path, P, off, cam, xy):
    P = np.ascontiguousarray(P, np.float64).reshape(-1, 12)
    nt = len(off) - 1
    with open(tmp_path / "in", "wb") as f:
        np.array([nt, len(P)], np.int64).tofile(f)
        P.tofile(f)
        np.asarray(off, np.int64).tofile(f)
        np.asarray(cam, np.uint32).tofile(f)
        np.asarray(xy, np.float64).reshape(-1, 2).tofile(f)
    subprocess.run([exe, str(tmp_path / "in"), str(tmp_path / "out")], check=True)
    o = np.fromfile(tmp_path / "out", np.float64)
    return o[:8 * nt].reshape(2, nt, 4), o[8 * nt:16 * nt].reshape(2, nt, 4), o[16 * nt:].reshape(2, nt) > 0


@pytest.mark.parametrize("pixels", [True, False])
@pytest.mark.parametrize("lens", [(2, 2), (3, 3), (2, 30)])
def test_short_form_matches_general(lens, pixels, exe, scenes, tmp_path):
    t = scenes.track_scene(num_cameras=60, num_tracks=20000, seed=sum(lens), min_len=lens[0], max_len=lens[1])
    P, xy = t["P"].reshape(-1, 3, 4), t["xy"]
    if not pixels:  # normalised image coordinates
        Ki = np.linalg.inv(np.array([[1000.0, 0, 960], [0, 1000, 540], [0, 0, 1]]))
        P, xy = Ki @ P, (np.concatenate([xy, np.ones((len(xy), 1))], 1) @ Ki.T)[:, :2]
    general, short, taken = run(exe, tmp_path, P, t["track_offsets"], t["camera_index"], xy)
    assert (taken.mean(1) > 0.99).all()
    for m in range(2):
        assert np.abs(general[m][taken[m]] - short[m][taken[m]]).max() < 1e-11


def test_degenerate_tracks(exe, scenes, tmp_path):
    t = scenes.track_scene(num_cameras=10, num_tracks=4, seed=3, min_len=3, max_len=3)
    # no view, one view, the same view three times, and 400 px of noise
    off = [0, 0, 1, 4, 7, 10]
    cam = np.concatenate([[0], [2, 2, 2], t["camera_index"][:3], t["camera_index"][3:6]])
    xy = np.concatenate([t["xy"][:1], np.repeat(t["xy"][1:2], 3, 0), t["xy"][:3], t["xy"][3:6] + [[400, -400]] * 3])
    general, short, taken = run(exe, tmp_path, t["P"], off, cam, xy)
    assert not taken[:, 0].any() and not taken[:, 1].any()
    for m in range(2):
        for k in range(2, 5):
            assert not taken[m, k] or np.abs(general[m, k] - short[m, k]).max() < 1e-11

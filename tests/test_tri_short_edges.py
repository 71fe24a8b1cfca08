"""Tracks that the FP64 estimators' short form has to leave to the general one,
on the CPU.  Without a single smallest direction (one view, the same view again,
cameras of one centre and exact images) any vector of a nullspace serves and
the general form's is kept: such tracks come back untaken.  With cameras of
very different scale the vector has the general form's sign and, where it is
taken, its accuracy: views at most 2^6 apart cost reflections at most 2^6
roundings (7e-15), the general form is within 1e-14 of the exact vector, so the
two differ by less than 2e-14."""
import numpy as np
import pytest

from test_tri_short_host import exe, run  # noqa: F401 (exe is a fixture)


def tracks(scenes, seed, count=4000, lo=2, hi=6):
    t = scenes.track_scene(num_cameras=60, num_tracks=count, seed=seed, min_len=lo, max_len=hi)
    return t["P"].reshape(-1, 3, 4), t["track_offsets"], t["camera_index"], t["xy"]


def image(P, cam, X):
    h = np.einsum("nij,nj->ni", P[cam], np.concatenate([X, np.ones((len(X), 1))], 1))
    return h[:, :2] / h[:, 2:]


@pytest.mark.parametrize("kind", ["one view", "repeated view", "one centre"])
def test_tracks_without_a_single_direction_are_left(kind, exe, scenes, tmp_path):  # noqa: F811
    n = 3000
    rng = np.random.default_rng(17)
    P = tracks(scenes, 5, count=10)[0]
    cam, xy = rng.integers(0, 60, n), rng.uniform(0, 1000, (n, 2))
    if kind == "one view":
        off = np.arange(n + 1)
    else:
        off, cam = 2 * np.arange(n + 1), np.repeat(cam, 2)
        xy = np.repeat(xy, 2, 0)
    if kind == "one centre":
        K = np.array([[1000.0, 0, 960], [0, 1000, 540], [0, 0, 1]])
        C = np.array([1.0, 2.0, -5.0])
        P = np.stack([K @ np.c_[R, -R @ C] for R in scenes.angle_axis_to_rotation(rng.normal(size=(60, 3)) * 0.1)])
        cam = rng.integers(0, 60, 2 * n)
        xy = image(P, cam, np.repeat(rng.uniform(-2, 2, (n, 3)) + [0, 0, 10], 2, 0))
    _, _, taken = run(exe, tmp_path, P, off, cam, xy)
    assert not taken.any()


@pytest.mark.parametrize("spread", [0, 1, 4, 8, 16])
def test_scaled_cameras_keep_sign_and_accuracy(spread, exe, scenes, tmp_path):  # noqa: F811
    P, off, cam, xy = tracks(scenes, 5)
    scale = 10.0 ** np.random.default_rng(spread).uniform(-spread / 2, spread / 2, (60, 1, 1))
    general, short, taken = run(exe, tmp_path, P * scale, off, cam, xy)
    if spread <= 1:
        assert (taken.mean(1) > 0.99).all()
    assert np.abs(general[1][taken[1]] - short[1][taken[1]]).max() < 2e-14
    # N-view: its design also has the images' size, about 1e3, in it
    assert np.abs(general[0][taken[0]] - short[0][taken[0]]).max() < 1e-11

"""A reduced system with pivots that are exactly zero.  A held camera at the
origin sees points on its axis only, at the principal point, so the columns of
its focal length and distortion are zero, and with no least LM diagonal so are
their rows of S, whatever the radius: every factorisation meets a zero pivot, in
the first tile, a middle one or the last.  No step can be taken: after the
allowed number of invalid steps the solve fails and the parameters keep their
bits.  With the usual least diagonal the same problem is solved."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def axis_scene(scenes, cameras, c, seed):
    sc = scenes.medium_scene(num_cameras=cameras, num_points=40 * cameras, mean_views=4, seed=seed,
                             hold=(0 if c else 1, c))
    rng = np.random.default_rng(seed)
    keep = sc["camera_index"] != c
    for f in ("observations", "camera_index", "intrinsic_index", "point_index"):
        sc[f] = sc[f][keep]
    sc["extrinsics"][c] = 0.0
    pp = sc["intrinsics"][c, 1:3]
    z = np.linspace(0.5, 3.0, 6)
    first = len(sc["points"])
    sc["points"] = np.concatenate([sc["points"], np.stack([0 * z, 0 * z, z], 1)])
    for q in (c, (c + 2) % cameras, (c + 3) % cameras):
        sc["observations"] = np.concatenate([sc["observations"], pp + rng.normal(0, 0.5 if q == c else 20.0, (6, 2))])
        sc["camera_index"] = np.append(sc["camera_index"], np.full(6, q)).astype(np.uint32)
        sc["intrinsic_index"] = np.append(sc["intrinsic_index"], np.full(6, q)).astype(np.uint32)
        sc["point_index"] = np.append(sc["point_index"], first + np.arange(6)).astype(np.uint32)
    return sc


# the camera's intrinsics at columns 36 of 84, 180 of 252 and 246 of 252
@pytest.mark.parametrize("cameras,c", [(8, 0), (22, 10), (22, 21)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_zero_pivots_stop_every_step(precision, cameras, c, handle, abi, scenes):
    sc = axis_scene(scenes, cameras, c, 400 + c)
    p = abi.PRECISION_MIXED if precision == "mixed" else abi.PRECISION_FP64
    opts = scenes.ba_options_for(sc, max_num_iterations=20, min_lm_diagonal=0.0, precision=p, fp64_polish_iterations=0)
    hp = abi.HostProblem(sc)
    before = hp.params()
    s = handle.solve(hp, opts)
    assert s.reduced_system_size == 12 * cameras - 12
    assert s.num_successful_steps == 0 and s.termination_type == abi.FAILURE and not s.usable
    assert s.final_cost == s.initial_cost
    for f, v in hp.params().items():
        np.testing.assert_array_equal(v, before[f])
    opts = scenes.ba_options_for(sc, max_num_iterations=5, precision=p, fp64_polish_iterations=0)
    s = handle.solve(abi.HostProblem(sc), opts)
    assert s.usable and s.num_successful_steps > 0 and s.final_cost < s.initial_cost

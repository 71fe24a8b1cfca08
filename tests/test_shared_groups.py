"""Free intrinsic groups shared by several cameras: the sums over points and
groups (k_group_*) against the point-major build, from which they differ by
the order of FP64 sums: the tolerances of the comparison of the camera-pair and
the point-major build.  One group, several, as many as the rule's mask holds, a
private and a held one among them, held coordinates, and points with more than
32 observations and with two of one camera; FP32 by a first step whose cost
keeps 1e-2 of the decrease (FP32 rounding times a condition of 1e5)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def shared_scene(scenes, model, groups, cameras=14, points=500, views=5):
    sc = scenes.medium_scene(num_cameras=cameras, num_points=points, mean_views=views, seed=500 + groups,
                             model=max(model, 1), hold=(0, 1), k_sigma=(0.05, 0.01, 0.01) if model else (0, 0, 0))
    if model == 0:  # without distortion and principal point
        sc["model"] = 0
        sc["observations"] = sc["observations"] - sc["intrinsics"][0, 1:3]
        sc["intrinsics"] = sc["intrinsics"][:, :1]
    sc["intrinsic_index"] = (sc["camera_index"] % groups).astype(np.uint32)
    sc["intrinsics"] = np.repeat(sc["intrinsics"][:1], groups, 0)
    return sc


def both(handle, abi, scenes, sc, **kw):
    out = []
    for build in (abi.SCHUR_BUILD_AUTO, abi.SCHUR_BUILD_POINT_ATOMIC):
        hp = abi.HostProblem(sc)
        opts = scenes.ba_options_for(sc, **kw)
        opts.schur_build = build
        out.append((handle.solve(hp, opts), hp))
    return out


@pytest.mark.parametrize("model", [0, 1, 2])
@pytest.mark.parametrize("groups,kind", [(1, ""), (2, ""), (3, "held"), (13, "private"), (4, "mask"), (2, "long"),
                                         (1, "twice")])
def test_matches_point_major_build(model, groups, kind, handle, abi, scenes):
    sc = shared_scene(scenes, model, groups, cameras=45 if kind == "long" else 14, views=40 if kind == "long" else 5,
                      points=150 if kind == "long" else 500)
    if kind == "held":
        sc["intrinsic_constant"] = np.array([0, 1, 0], np.uint8)
    if kind == "mask":
        sc["extrinsic_fixed_mask"] = 0b100001
        sc["intrinsic_fixed_mask"] = 0b110 if model else 0
    if kind == "twice":  # every fifth observation again, half a pixel off
        for k in ("observations", "camera_index", "intrinsic_index", "point_index"):
            sc[k] = np.concatenate([sc[k], sc[k][::5] + (0.5 if k == "observations" else 0)]).astype(sc[k].dtype)
    (a, ha), (b, hb) = both(handle, abi, scenes, sc, max_num_iterations=4)
    assert a.usable and a.num_iterations == b.num_iterations and a.reduced_system_size == b.reduced_system_size
    assert abs(a.final_cost - b.final_cost) <= 1e-10 * b.final_cost
    for f in ("extrinsics", "points"):
        np.testing.assert_allclose(getattr(ha, f), getattr(hb, f), rtol=0, atol=1e-8)
    x, y = ha.intrinsics, hb.intrinsics
    np.testing.assert_allclose(x, y, rtol=0, atol=1e-8 * np.abs(y).max())
    (c, hc), _ = both(handle, abi, scenes, sc, max_num_iterations=4)
    assert np.array_equal(ha.points, hc.points) and a.final_cost == c.final_cost  # no atomics: repeatable


def test_camera_of_several_groups_keeps_the_point_major_build(handle, abi, scenes):
    sc = shared_scene(scenes, 1, 2)
    sc["intrinsic_index"][::3] ^= 1
    (a, ha), (b, hb) = both(handle, abi, scenes, sc, max_num_iterations=3)
    assert a.usable and abs(a.final_cost - b.final_cost) <= 1e-10 * b.final_cost
    np.testing.assert_allclose(ha.points, hb.points, rtol=0, atol=1e-8)


@pytest.mark.parametrize("groups", [1, 3])
def test_mixed_first_step(groups, handle, abi, scenes):
    sc = shared_scene(scenes, 1, groups)
    (d, _), _ = both(handle, abi, scenes, sc, max_num_iterations=1)
    (f, _), _ = both(handle, abi, scenes, sc, max_num_iterations=1, precision=abi.PRECISION_MIXED)
    assert d.num_successful_steps == f.num_successful_steps == 1
    assert abs(f.final_cost - d.final_cost) <= 1e-2 * (d.initial_cost - d.final_cost)

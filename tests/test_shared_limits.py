"""Shared intrinsic groups beyond what the camera-pair list can hold: more pairs
than its 32-bit sort counts, or no device memory for it.  Both are solved by the
point-major build, with the result that the option for that build gives, up to
the order of its atomic sums (the tolerances of the other comparisons)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def all_seen(scenes, cameras, points, seed):
    """Every camera sees every point, one pinhole group for all."""
    sc = scenes.medium_scene(num_cameras=cameras, num_points=points, mean_views=1, seed=seed, hold=(0, 1),
                             k_sigma=(0, 0, 0), sigma=0.0, outlier_frac=0.0)
    rng = np.random.default_rng(seed)
    ext, X = sc["extrinsics"].reshape(-1, 6), sc["points"].reshape(-1, 3)
    R = scenes.angle_axis_to_rotation(ext[:, :3])
    p = np.einsum("nij,mj->mni", R, X) + ext[None, :, 3:]
    obs = 1000.0 * p[..., :2] / p[..., 2:] + rng.normal(0, 0.7, p.shape[:2] + (2,))
    n = points * cameras
    return dict(model=0, extrinsics=ext, intrinsics=np.full((1, 1), 1003.0), points=X + rng.normal(0, 0.01, X.shape),
                observations=obs.reshape(n, 2), camera_index=np.tile(np.arange(cameras), points).astype(np.uint32),
                intrinsic_index=np.zeros(n, np.uint32),
                point_index=np.repeat(np.arange(points), cameras).astype(np.uint32),
                camera_constant=sc["camera_constant"])


def solve(h, abi, sc, build, iterations):
    hp = abi.HostProblem(sc)
    s = h.solve(hp, abi.default_options(max_num_iterations=iterations, schur_build=build))
    return s, hp


def same(a, b):
    (sa, ha), (sb, hb) = a, b
    assert sa.usable and sa.num_successful_steps > 0 and sa.num_iterations == sb.num_iterations
    assert abs(sa.final_cost - sb.final_cost) <= 1e-9 * sb.final_cost
    np.testing.assert_allclose(ha.points, hb.points, rtol=0, atol=1e-8)
    np.testing.assert_allclose(ha.intrinsics, hb.intrinsics, rtol=1e-9)


def test_more_pairs_than_the_list_counts(gb, abi, scenes):
    cameras, points = 1000, 4300
    assert points * cameras * (cameras + 1) // 2 > 0x7fffffff
    sc = all_seen(scenes, cameras, points, 951)
    h = gb.Handle(0)
    try:
        same(solve(h, abi, sc, abi.SCHUR_BUILD_AUTO, 1), solve(h, abi, sc, abi.SCHUR_BUILD_POINT_ATOMIC, 1))
    finally:
        h.close()


def test_no_memory_for_the_list(gb, abi, scenes):
    import torch
    sc = all_seen(scenes, 200, 1500, 952)
    pairs = 1500 * 200 * 201 // 2
    ref = gb.Handle(0)
    full = solve(ref, abi, sc, abi.SCHUR_BUILD_AUTO, 3)
    ref.close()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    # room for the records (71 values an observation) and the workspace, not
    # for the list (28 bytes a pair and its sort's workspace)
    room = 700 << 20
    assert 300000 * 71 * 8 + (200 << 20) < room < 300000 * 71 * 8 + 28 * pairs
    free = torch.cuda.mem_get_info()[0]
    rest = torch.empty(free - room, dtype=torch.uint8, device="cuda:0")
    h = gb.Handle(0)
    try:
        small = solve(h, abi, sc, abi.SCHUR_BUILD_AUTO, 3)
    finally:
        h.close()
        del rest
        torch.cuda.empty_cache()
    same(small, full)

"""Backward substitution by 16-column blocks (up to 8 tiles of 64) and by the
tiles' inverses (beyond), at the last sizes of one and the first of the other
and inside the first tile, against the oracle with the tolerances of the other
FP64 comparisons: costs 1e-9 relative, points 1e-8."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 12 columns a camera, two held extrinsics: 24, 60, 72 columns, 504 (8 tiles), 516 and 528 (9)
@pytest.mark.parametrize("cameras", [3, 6, 7, 43, 44, 45])
def test_both_sides_of_the_rule(cameras, handle, abi, scenes, oracle_mod):
    sc = scenes.medium_scene(num_cameras=cameras, num_points=40 * cameras, mean_views=min(5, cameras - 2),
                             seed=350 + cameras, hold=(0, 1))
    opts = scenes.ba_options_for(sc, max_num_iterations=3)
    hp = abi.HostProblem(sc)
    s = handle.solve(hp, opts)
    _, so, po, _ = oracle_mod.ba_solve(sc, opts)
    assert s.usable and s.reduced_system_size == 12 * cameras - 12 and s.num_iterations == so["num_iterations"]
    assert abs(s.final_cost - so["final_cost"]) <= 1e-9 * so["final_cost"]
    np.testing.assert_allclose(hp.points.reshape(-1, 3), np.asarray(po["points"]).reshape(-1, 3), rtol=0, atol=1e-8)

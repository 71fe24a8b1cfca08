"""Dense factorisation, FP64 (panels on the FP64 pipe, trailing update by exact
FP16 digit products on the tensor cores): reduced systems on both sides of its
16-column blocks, 64-column panels and 128-row tile pairs, and one with
several panels of look-ahead, against the CPU oracle.  The step solves a
system of condition up to about 1e6 in FP64 arithmetic, so the parameters
after a few iterations agree to 1e-8 and the costs to 1e-9 relative, the
tolerances of the other FP64 comparisons with the oracle.  The FP32
factorisation of the mixed path is checked on the same sizes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# cameras with 12 (radial K3) or 14 (Brown-T2) columns each, two held extrinsics
@pytest.mark.parametrize("model,cameras", [(1, 3), (1, 6), (2, 6), (1, 11), (1, 12), (2, 10), (1, 17), (1, 22), (1, 45)])
def test_panel_edges_match_oracle(model, cameras, handle, abi, scenes, oracle_mod):
    sc = scenes.medium_scene(num_cameras=cameras, num_points=40 * cameras, mean_views=min(5, cameras - 2),
                             seed=300 + cameras, model=model, hold=(0, 1))
    opts = scenes.ba_options_for(sc, max_num_iterations=3)
    hp = abi.HostProblem(sc)
    s = handle.solve(hp, opts)
    _, so, po, _ = oracle_mod.ba_solve(sc, opts)
    assert s.usable and s.num_iterations == so["num_iterations"]
    assert abs(s.final_cost - so["final_cost"]) <= 1e-9 * so["final_cost"]
    np.testing.assert_allclose(hp.points.reshape(-1, 3), np.asarray(po["points"]).reshape(-1, 3), rtol=0, atol=1e-8)


@pytest.mark.parametrize("cameras", [6, 11, 12, 17, 22, 45])
def test_mixed_panel_edges_step_as_fp64(cameras, handle, abi, scenes):
    """The FP32 panel and TF32 trailing update on the same sizes, one LM step.
    With a relative error of the step of at most 1e-2 (FP32 rounding times a
    condition of 1e5) the cost after it differs from the FP64 step's by at
    most that share of the decrease; a wrong tile or digit misses the descent
    altogether."""
    sc = scenes.medium_scene(num_cameras=cameras, num_points=40 * cameras, mean_views=min(5, cameras - 2),
                             seed=330 + cameras, hold=(0, 1))
    end = {}
    for p in (abi.PRECISION_FP64, abi.PRECISION_MIXED):
        s = handle.solve(abi.HostProblem(sc), scenes.ba_options_for(sc, max_num_iterations=1, precision=p))
        assert s.usable and s.num_successful_steps == 1
        start, end[p] = s.initial_cost, s.final_cost
    drop = start - end[abi.PRECISION_FP64]
    assert abs(end[abi.PRECISION_MIXED] - end[abi.PRECISION_FP64]) <= 1e-2 * drop


def test_indefinite_system_is_rejected(handle, abi, scenes):
    """A camera block that is not positive definite (a zero LM diagonal and a
    camera without a second observation) fails its pivot: the step is invalid
    or rejected, and the parameters stay finite."""
    sc = scenes.medium_scene(num_cameras=8, num_points=60, mean_views=2, seed=311)
    opts = scenes.ba_options_for(sc, max_num_iterations=4, min_lm_diagonal=0.0, max_lm_diagonal=0.0)
    hp = abi.HostProblem(sc)
    s = handle.solve(hp, opts)
    assert np.isfinite(hp.points).all() and np.isfinite(hp.extrinsics).all()
    assert s.final_cost <= s.initial_cost

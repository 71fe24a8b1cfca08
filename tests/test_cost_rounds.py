"""The cost pass deals the outliers of four observations a thread to the lanes
of their warp, and the point kernels deal a group's FP64 work to theirs: costs
at the edges of a round (none, some and all outliers) against the oracle, FP64
sums of the same terms in another order, 1e-12; and the first step with points
of two observations (16 points a group, two rounds) or one, whose cost keeps
1e-2 of the FP64 step's decrease (FP32 rounding times a condition of 1e5; a
radius of 1, since an undamped first step fails on weakly observed points)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("scale", [1e-6, 1.0, 1e6])
@pytest.mark.parametrize("count", [1, 31, 33, 127, 1025, 16384, 20001])
def test_cost_at_the_edges_of_a_round(count, scale, mixed, handle, abi, scenes, oracle_mod):
    sc = scenes.medium_scene(num_cameras=12, num_points=4000, mean_views=5, seed=81, hold=(0, 1))
    assert len(sc["observations"]) >= count
    for k in ("observations", "camera_index", "intrinsic_index", "point_index"):
        sc[k] = sc[k][:count]
    sc["loss"], sc["loss_scale"] = abi.LOSS_HUBER, scale
    s = handle.solve(abi.HostProblem(sc), scenes.ba_options_for(
        sc, max_num_iterations=0, fp64_polish_iterations=0,
        precision=abi.PRECISION_MIXED if mixed else abi.PRECISION_FP64))
    ref = oracle_mod.ba_evaluate(sc, abi.LOSS_HUBER, scale)["cost"]
    assert abs(s.initial_cost - ref) <= 1e-12 * ref


@pytest.mark.parametrize("solver", ["dense", "pcg"])
@pytest.mark.parametrize("views", [1, 2])
def test_groups_of_many_points(views, solver, handle, abi, scenes):
    sc = scenes.medium_scene(num_cameras=12, num_points=1500, mean_views=5, seed=82, hold=(0, 1))
    # the last 500 points keep `views` observations
    seen = np.zeros(1500, int)
    keep = np.ones(len(sc["point_index"]), bool)
    for i, p in enumerate(sc["point_index"]):
        seen[p] += 1
        keep[i] = p < 1000 or seen[p] <= views
    for k in ("observations", "camera_index", "intrinsic_index", "point_index"):
        sc[k] = sc[k][keep]
    end = {}
    for p in (abi.PRECISION_FP64, abi.PRECISION_MIXED):
        o = scenes.ba_options_for(sc, max_num_iterations=1, precision=p, fp64_polish_iterations=0,
                                  initial_trust_region_radius=1.0)
        if solver == "pcg":
            o.linear_solver = abi.SOLVER_ITERATIVE_SCHUR
        s = handle.solve(abi.HostProblem(sc), o)
        assert s.usable and s.num_successful_steps == 1
        start, end[p] = s.initial_cost, s.final_cost
    assert abs(end[abi.PRECISION_MIXED] - end[abi.PRECISION_FP64]) <= 1e-2 * (start - end[abi.PRECISION_FP64])

"""Counts of runs and sums of groups inside a warp: observations point by point,
shuffled, alternating between two points and all of one point, with few and
many intrinsic groups, give the same solve but for the order of observations
inside a point (the tolerance of the comparison of shuffled observations), and
an index out of range anywhere is refused."""
import numpy as np
import pytest

from test_shared_groups import shared_scene

pytestmark = pytest.mark.gpu
FIELDS = ("observations", "camera_index", "intrinsic_index", "point_index")


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("groups", [1, 3, 14, 70])
@pytest.mark.parametrize("order", ["points", "shuffled", "cameras", "striped"])
def test_any_order_gives_the_same_cost(order, groups, mixed, handle, abi, scenes):
    sc = shared_scene(scenes, 1, groups, cameras=80 if groups == 70 else 14)
    o = scenes.ba_options_for(sc, max_num_iterations=1, fp64_polish_iterations=0,
                              precision=abi.PRECISION_MIXED if mixed else abi.PRECISION_FP64)
    a = handle.solve(abi.HostProblem(sc), o)
    n = len(sc["point_index"])
    at = {"points": np.argsort(sc["point_index"], kind="stable"), "shuffled": np.random.default_rng(4).permutation(n),
          "cameras": np.argsort(sc["camera_index"], kind="stable"),
          "striped": np.arange(n).reshape(2, -1).T.ravel() if n % 2 == 0 else np.r_[np.arange(n - 1).reshape(2, -1).T.ravel(), n - 1]}
    for k in FIELDS:
        sc[k] = sc[k][at[order]]
    b = handle.solve(abi.HostProblem(sc), o)
    assert a.usable and a.num_successful_steps == b.num_successful_steps
    # FP32: the step's rounding, as 1e-2 of the decrease
    tol = 1e-2 * (a.initial_cost - a.final_cost) if mixed else 1e-9 * a.final_cost
    assert abs(a.final_cost - b.final_cost) <= tol and abs(a.initial_cost - b.initial_cost) <= 1e-12 * a.initial_cost


@pytest.mark.parametrize("at", [0, 5, 31, 32, -1])
@pytest.mark.parametrize("field", ["camera_index", "intrinsic_index", "point_index"])
def test_index_out_of_range_is_refused(field, at, handle, abi, scenes):
    import ctypes as C
    sc = shared_scene(scenes, 1, 2)
    sc[field] = sc[field].copy()
    sc[field][at] = 10 ** 6
    hp = abi.HostProblem(sc)
    p, s = hp.struct(), abi.GbbaSummary()
    st = handle.lib.gbba_solve(handle.h, C.byref(p), C.byref(abi.default_options()), C.byref(s))
    assert st == abi.ERROR_INVALID_ARGUMENT

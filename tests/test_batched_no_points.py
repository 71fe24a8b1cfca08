"""Windows without points: observations of a point that is not there are an
index out of range, whether the batch has other points or none."""
import numpy as np
import pytest

from test_ba_gpu import batched_solve, local_problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("windows", [1, 2, 40])
@pytest.mark.parametrize("others", [0, 1])
def test_observations_without_points_are_refused(windows, others, precision, handle, abi, scenes):
    o = abi.default_options(precision=abi.PRECISION_MIXED if precision == "mixed" else abi.PRECISION_FP64)
    probs = local_problems(scenes, windows, seed=921, cams=(5, 6), points=(20, 30))
    none = [dict(p, points=np.zeros((0, 3))) for p in probs]
    st, s, prm = batched_solve(handle, abi, none + probs[:others], o)
    assert st == abi.ERROR_INVALID_ARGUMENT
    for p, q in zip(none + probs[:others], prm):
        np.testing.assert_array_equal(np.ravel(p["extrinsics"]), np.ravel(q["extrinsics"]))

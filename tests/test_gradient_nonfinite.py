"""Gradients of observations that are not finite: a NaN or infinite residual
makes every term J^T r of its camera, group and point non-finite, also where
the Jacobian entry is small or zero (0 * NaN is NaN), so those entries are NaN
and no others change by a bit."""
import ctypes as C

import numpy as np
import pytest

from test_camera_lin import scene

pytestmark = pytest.mark.gpu


def gradients(handle, abi, sc, loss, mixed):
    """From the stored blocks and from blocks evaluated again."""
    p = (hp := abi.HostProblem(sc)).struct()
    no, k = p.num_observations, abi.MODEL_K[hp.model]
    fn = handle.lib.gbba_project_backward_mixed if mixed else handle.lib.gbba_project_backward
    je, jk, jx = np.zeros((no, 12)), np.zeros((no, 2 * k)), np.zeros((no, 6))
    out = []
    for blocks in ([je, jk, jx], [None] * 3):
        g = np.zeros(6 * p.num_cameras + k * p.num_intrinsics + 3 * p.num_points)
        handle.check(fn(handle.h, C.byref(p), loss, 4.0, *[b.ctypes.data if b is not None else None for b in blocks],
                        g.ctypes.data), "backward")
        out.append(g)
    return out


@pytest.mark.parametrize("model", [0, 1, 2])
@pytest.mark.parametrize("loss", [0, 1])
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("axis", [0, 1])
def test_touched_entries_are_nan(model, loss, mixed, value, axis, handle, abi, scenes):
    sc = scene(scenes, abi, model)
    ref = gradients(handle, abi, sc, loss, mixed)
    at = 29
    sc["observations"] = sc["observations"].copy()
    sc["observations"][at, axis] = value
    c, p, k = int(sc["camera_index"][at]), int(sc["point_index"][at]), abi.MODEL_K[model]
    nc, ng = len(sc["extrinsics"]), len(sc["intrinsics"])
    touched = np.zeros(len(ref[0]), bool)
    touched[6 * c:6 * c + 6] = True
    touched[6 * nc + k * c:6 * nc + k * c + k] = True  # a group per camera
    touched[6 * nc + k * ng + 3 * p:][:3] = True
    for g, r in zip(gradients(handle, abi, sc, loss, mixed), ref):
        assert np.isnan(g[touched]).all() and np.isfinite(r).all()
        np.testing.assert_array_equal(g[~touched], r[~touched])

"""FP64 Jacobians from the cameras' linearisation data: rotations on both sides
of the first-order branch, small ones (where 1 - cos cancels), half turns and
beyond, for every camera model, against the oracle's AutoDiff.  Both evaluate
the same derivative in FP64 from values up to about 1e4: 1e-9 relative to a
block's largest entry, the bound of the other AutoDiff comparisons, and for a
small angle th the rounding of AutoDiff's own 1 / th terms, 1e-15 / th (6e-8 at
the smallest, hence the gradient's 1e-7).  The gradient summed from the stored blocks equals, bit for bit, the one summed
from blocks evaluated again, and a parameter without observations gets 0."""
import ctypes as C

import numpy as np
import pytest

from test_ba_gpu import project

pytestmark = pytest.mark.gpu

ANGLES = [0.0, 1e-9, 1.4e-8, 1.6e-8, 1e-6, 1e-4, 1e-2, 1.0, 3.0, np.pi, 4.0]


def scene(scenes, abi, model):
    sc = scenes.ring_scene(num_cameras=4, num_points=12, seed=61, model=model) if model == 0 else \
        scenes.medium_scene(num_cameras=4, num_points=12, seed=61 + model, model=model)
    # cameras of the given angles in front of points around (0, 0, 8) of their frame
    rng = np.random.default_rng(3)
    n = len(ANGLES)
    axis = rng.normal(size=(n, 3))
    axis /= np.linalg.norm(axis, axis=1)[:, None]
    ext = np.concatenate([axis * np.array(ANGLES)[:, None], np.zeros((n, 3))], 1)
    R = scenes.angle_axis_to_rotation(ext[:, :3])
    X = rng.uniform(-1, 1, (12, 3))
    ext[:, 3:] = [0.1, -0.2, 8.0]
    cam = np.repeat(np.arange(n), 12).astype(np.uint32)
    pt = np.tile(np.arange(12), n).astype(np.uint32)
    intr = np.repeat(sc["intrinsics"][:1], n, 0)
    assert (np.einsum("nij,mj->nmi", R, X)[..., 2] + 8.0 > 5).all()
    return dict(model=model, extrinsics=ext, intrinsics=intr, points=X, observations=rng.normal(size=(12 * n, 2)) * 50,
                camera_index=cam, intrinsic_index=cam.copy(), point_index=pt)


@pytest.mark.parametrize("model", [0, 1, 2])
def test_blocks_match_autodiff(model, handle, abi, scenes, oracle_mod):
    sc = scene(scenes, abi, model)
    ev = project(handle, abi, sc, abi.LOSS_HUBER, 4.0)
    ref = oracle_mod.ba_evaluate(sc, abi.LOSS_HUBER, 4.0)
    for k in ("jac_extrinsic", "jac_intrinsic", "jac_point"):
        a, b = ev[k].reshape(len(ANGLES), -1), np.asarray(ref[k]).reshape(len(ANGLES), -1)
        for i, th in enumerate(ANGLES):
            tol = 1e-9 + (1e-15 / th if th > 1.5e-8 else 0.0)
            np.testing.assert_allclose(a[i], b[i], rtol=0, atol=tol * np.abs(b).max())
    np.testing.assert_allclose(ev["gradient"], ref["gradient"], rtol=0, atol=1e-7 * np.abs(ref["gradient"]).max())


@pytest.mark.parametrize("model", [0, 1, 2])
@pytest.mark.parametrize("mixed", [False, True])
def test_gradient_routes_agree(model, mixed, handle, abi, scenes):
    sc = scene(scenes, abi, model)
    sc["points"] = np.concatenate([sc["points"], np.ones((3, 3))])  # three points without observations
    full = project(handle, abi, sc, abi.LOSS_HUBER, 4.0, mixed=mixed)["gradient"]
    hp = abi.HostProblem(sc)
    p = hp.struct()
    g = np.full_like(full, np.nan)
    fn = handle.lib.gbba_project_backward_mixed if mixed else handle.lib.gbba_project_backward
    handle.check(fn(handle.h, C.byref(p), abi.LOSS_HUBER, 4.0, None, None, None, g.ctypes.data), "backward")
    np.testing.assert_array_equal(g, full)
    assert (full[-9:] == 0).all() and np.isfinite(full).all()


@pytest.mark.parametrize("cut", [1, 0, -1])
def test_solver_on_both_sides_of_the_rule(cut, handle, abi, scenes, oracle_mod):
    """16383, 16384 and 16385 observations (the solver takes the linearisation
    data from 16384 on) against the oracle's iterations, with the tolerances
    of the other FP64 comparisons."""
    sc = scenes.medium_scene(num_cameras=12, num_points=4000, mean_views=5, seed=71, hold=(0, 1))
    assert len(sc["observations"]) >= 16385
    for k in ("observations", "camera_index", "intrinsic_index", "point_index"):
        sc[k] = sc[k][:16384 - cut]
    opts = scenes.ba_options_for(sc, max_num_iterations=2)
    hp = abi.HostProblem(sc)
    s = handle.solve(hp, opts)
    _, so, po, _ = oracle_mod.ba_solve(sc, opts)
    assert s.usable and s.num_iterations == so["num_iterations"]
    assert abs(s.final_cost - so["final_cost"]) <= 1e-9 * so["final_cost"]
    np.testing.assert_allclose(hp.extrinsics.reshape(-1, 6), np.asarray(po["extrinsics"]).reshape(-1, 6), rtol=0,
                               atol=1e-8)

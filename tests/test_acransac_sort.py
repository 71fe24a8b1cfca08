"""gbsfm_acransac_score on both sides of each sort size (256 to 8,192 pairs and
the global slice above), with ties that the sort's 51 error bits cannot tell
apart (repeated correspondences) and models without a finite error, against
the C++ oracle: order, inlier counts and thresholds exact, NFA to the tables'
float rounding (the tolerances of the fixture comparisons)."""
import math

import numpy as np
import pytest

from test_sfm_acransac import NFA_TOL, gpu_score

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [7, 8, 255, 256, 257, 512, 513, 1024, 1025, 2047, 2048, 2049, 4096, 4097, 8191, 8192, 8193])
def test_sort_sizes_and_ties(n, handle, abi, scenes, oracle_mod):
    sc = scenes.resection_scene(num_points=n, seed=n)
    rng = np.random.default_rng(n)
    x = (sc["x2d"] - np.array([960.0, 540.0])) / 1000.0
    X = sc["x3d"].copy()
    same = rng.integers(0, n, n // 3)  # a third repeats another correspondence
    x[:len(same)], X[:len(same)] = x[same], X[same]
    R = np.array([[1.0, 0, 0, 0.1], [0, 1, 0, -0.2], [0, 0, 1, 8.0]])
    models = np.stack([R * (1 + 0.01 * rng.normal(size=(3, 4))) for _ in range(12)]).reshape(-1, 12)
    models[3] = 0.0  # every error is not a number
    for thr in (math.inf, 1e-3):
        st, (nfa, k, emax, order) = gpu_score(handle, abi, x, X, models, 6, 1, math.log10(math.pi), max_threshold=thr)
        handle.check(st, "gbsfm_acransac_score")
        rn, rk, re, ro, _ = oracle_mod.acransac_score_cpp(x, X, models, 6, 1, math.log10(math.pi), max_threshold=thr)
        np.testing.assert_array_equal(k, rk)
        ok = np.isfinite(rn)
        np.testing.assert_array_equal(ok, np.isfinite(nfa))
        np.testing.assert_allclose(nfa[ok], rn[ok], rtol=0, atol=NFA_TOL)
        np.testing.assert_allclose(emax[ok], re[ok], rtol=1e-12, atol=0)
        for m in range(len(models)):
            np.testing.assert_array_equal(np.sort(order[m]), np.arange(n))
            if m != 3:
                np.testing.assert_array_equal(order[m, :k[m]], ro[m, :rk[m]])

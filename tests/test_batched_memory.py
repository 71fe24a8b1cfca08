"""A batch whose windows would get four CTAs each where device memory holds the
scratch of one: it is solved with one, with the same bits (the sums of S are
integers).  One point with 4,000 observations makes the scratch large: 16 warps
times 4,001 slots of 1,344 bytes a CTA, 86 MB."""
import numpy as np
import pytest

from test_ba_gpu import batched_solve, local_problems

pytestmark = pytest.mark.gpu


def test_scratch_of_one_cta_is_enough(gb, abi, scenes):
    import torch
    probs = local_problems(scenes, 30, seed=971, cams=(5, 6), points=(60, 80))
    p = probs[0]
    at = int(np.flatnonzero(p["point_index"] == p["point_index"][0])[0])
    rng = np.random.default_rng(971)
    p["observations"] = np.concatenate([p["observations"].reshape(-1, 2),
                                        p["observations"].reshape(-1, 2)[at] + rng.normal(0, 0.5, (4000, 2))])
    for f in ("camera_index", "intrinsic_index", "point_index"):
        p[f] = np.concatenate([p[f], np.full(4000, p[f][at])]).astype(np.uint32)
    o = abi.default_options(precision=abi.PRECISION_MIXED, max_num_iterations=4, fp64_polish_iterations=0)
    one = 30 * 16 * 4001 * 1344
    runs = []
    for room in (None, 2 * one):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        rest = None
        if room:
            rest = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda:0")
        h = gb.Handle(0)
        try:
            runs.append(batched_solve(h, abi, probs, o))
        finally:
            h.close()
            del rest
            torch.cuda.empty_cache()
    (st, s, prm), (st1, s1, prm1) = runs
    assert st == st1 == abi.SUCCESS
    for a, b, x, y in zip(s, s1, prm, prm1):
        assert a.usable and a.final_cost == b.final_cost and a.num_iterations == b.num_iterations
        for f in ("extrinsics", "intrinsics", "points"):
            np.testing.assert_array_equal(x[f], y[f])

"""Windows built by one CTA against the same windows built by four: in a batch of
more windows than 76 only those of more than an SM's mean load get two CTAs, so
beside 200 larger ones the windows under test get one.  The sums of S are
integers, so the solve keeps its bits.  One intrinsic group and several, the
build's two forms."""
import numpy as np
import pytest

from test_ba_gpu import batched_solve, local_problems

pytestmark = pytest.mark.gpu


def load(p):  # the dispatch's measure: observations and their pairs
    o = len(p["camera_index"])
    return o * (12.0 + o / max(1, len(np.asarray(p["points"]).reshape(-1, 3))))


@pytest.mark.parametrize("groups", [1, 2])
def test_one_cta_gives_the_bits_of_four(groups, handle, abi, scenes):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    w = local_problems(scenes, 3, seed=941, cams=(5, 12), points=(100, 600))
    if groups == 2:
        for p in w:
            p["intrinsic_index"] = (p["camera_index"] % 2).astype(np.uint32)
            p["intrinsics"] = np.repeat(p["intrinsics"].reshape(-1, 8)[:1], 2, 0)
    fill = local_problems(scenes, 4, seed=942, cams=(16, 18), points=(1000, 1200)) * 50
    assert 4 * len(w) <= sms and 2 * (len(w) + len(fill)) > sms
    assert max(map(load, w)) < sum(map(load, w + fill)) / sms
    o = abi.default_options(precision=abi.PRECISION_MIXED, max_num_iterations=5, fp64_polish_iterations=0)
    st, s4, p4 = batched_solve(handle, abi, w, o)
    st1, s1, p1 = batched_solve(handle, abi, w + fill, o)
    assert st == st1 == abi.SUCCESS
    for i in range(3):
        assert s4[i].usable and s4[i].num_iterations == s1[i].num_iterations
        assert s4[i].final_cost == s1[i].final_cost
        for f in ("extrinsics", "intrinsics", "points"):
            np.testing.assert_array_equal(p4[i][f], p1[i][f])

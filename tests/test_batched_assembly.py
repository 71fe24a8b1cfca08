"""Assembly of a batch: a window's solve does not depend on the others, so
packed copies (small windows), copies per window (large ones) and device arrays
give the same bits, for observations in any order and windows without any."""
import ctypes as C

import numpy as np
import pytest

from test_ba_gpu import batched_solve, local_problems

pytestmark = pytest.mark.gpu


def large(scenes):
    # 3,000 points, 8 cameras and more: over 64 KB of each array but the cameras'
    return local_problems(scenes, 2, seed=901, cams=(8, 12), points=(3000, 3200))


def test_copies_per_window_and_packed_agree(handle, abi, scenes):
    o = abi.default_options(precision=abi.PRECISION_MIXED, max_num_iterations=3)
    big = large(scenes)
    small = local_problems(scenes, 40, seed=902, points=(50, 60))
    empty = dict(small[0], observations=np.zeros((0, 2)), camera_index=np.zeros(0, np.uint32),
                 intrinsic_index=np.zeros(0, np.uint32), point_index=np.zeros(0, np.uint32))
    for p in big:
        perm = np.random.default_rng(1).permutation(len(p["observations"]))
        for f in ("observations", "camera_index", "intrinsic_index", "point_index"):
            p[f] = p[f][perm]
    assert big[0]["camera_index"].size * 4 > 65536 > sum(p["camera_index"].size * 4 for p in big + small) / 43
    st, s1, p1 = batched_solve(handle, abi, big, o)
    st2, s2, p2 = batched_solve(handle, abi, [empty] + small + big, o)
    assert st == st2 == abi.SUCCESS and all(s.usable for s in s1 + s2)
    np.testing.assert_array_equal(p2[0]["points"], empty["points"])
    dev = [abi.DeviceProblem(p) for p in big]
    structs = (abi.GbbaProblem * 2)(*[d.struct() for d in dev])
    s3 = (abi.GbbaSummary * 2)()
    handle.check(handle.lib.gbba_solve_batched(handle.h, structs, 2, C.byref(o), s3), "batched")
    for i in range(2):
        assert s1[i].final_cost == s2[41 + i].final_cost == s3[i].final_cost
        for f in ("extrinsics", "intrinsics", "points"):
            np.testing.assert_array_equal(p1[i][f], p2[41 + i][f])
            np.testing.assert_array_equal(p1[i][f].ravel(), dev[i].params()[f].ravel())


@pytest.mark.parametrize("field,value", [("camera_index", 12), ("intrinsic_index", 1), ("point_index", 3200)])
def test_index_out_of_range_is_rejected(field, value, handle, abi, scenes):
    probs = large(scenes)
    probs[1][field] = probs[1][field].copy()
    probs[1][field][-1] = value
    before = [p["points"].copy() for p in probs]
    st, _, prm = batched_solve(handle, abi, probs, abi.default_options(precision=abi.PRECISION_MIXED))
    assert st == abi.ERROR_INVALID_ARGUMENT
    for a, b in zip(before, prm):
        np.testing.assert_array_equal(a, b["points"])

"""A window built by one, two or four CTAs: the shares of S are integer sums, so
its solve is the same bit for bit in batches that give it a different number
(up to 38 windows four CTAs each, up to 76 two, beyond that two for the large
ones and one for the others).  Windows with fewer points than warps leave
helpers without work; windows with several groups take the general build."""
import numpy as np
import pytest

from test_ba_gpu import batched_solve, local_problems

pytestmark = pytest.mark.gpu


def windows(scenes, kind):
    if kind == "few points":
        return local_problems(scenes, 3, seed=911, cams=(5, 6), points=(20, 33))
    out = local_problems(scenes, 3, seed=912, cams=(5, 14), points=(100, 700))
    if kind == "groups":
        for p in out:
            nc = p["extrinsics"].size // 6
            p["intrinsic_index"] = (p["camera_index"] % 2).astype(np.uint32)
            p["intrinsics"] = np.repeat(p["intrinsics"].reshape(-1, 8)[:1], 2, 0)
            assert nc > 2
    return out


@pytest.mark.parametrize("kind", ["one group", "groups", "few points"])
def test_any_number_of_ctas_gives_the_same_bits(kind, handle, abi, scenes):
    o = abi.default_options(precision=abi.PRECISION_MIXED, max_num_iterations=5, fp64_polish_iterations=0)
    w = windows(scenes, kind)
    fill = local_problems(scenes, 200, seed=913, cams=(5, 6), points=(60, 80))
    ref = None
    for extra in (0, 50, 200):
        st, s, p = batched_solve(handle, abi, w + fill[:extra], o)
        assert st == abi.SUCCESS
        s, p = s[:3], p[:3]
        if ref is None:
            ref = s, p
        for i in range(3):
            assert s[i].usable and s[i].final_cost == ref[0][i].final_cost
            assert s[i].num_iterations == ref[0][i].num_iterations
            for f in ("extrinsics", "intrinsics", "points"):
                np.testing.assert_array_equal(p[i][f], ref[1][i][f])


def test_nonfinite_window_releases_its_helpers(handle, abi, scenes):
    w = windows(scenes, "one group")
    w[1]["observations"] = w[1]["observations"].copy()
    w[1]["observations"].reshape(-1)[3] = np.nan
    st, s, _ = batched_solve(handle, abi, w, abi.default_options(precision=abi.PRECISION_MIXED,
                                                                 fp64_polish_iterations=0))
    assert st == abi.ERROR_NUMERICAL and s[0].usable and not s[1].usable and s[2].usable

"""gbsfm_pack_ba around its tile and chunk edges: entry counts at multiples of
the 2,048-entry tile and one off, runs of empty tracks across a tile edge, one
track longer than a tile, and image counts on both sides of a block and of the
8,192-image chunk of the ordinals, against a numpy restatement (exact)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def state(lens, num_images, seed):
    rng = np.random.default_rng(seed)
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    ne, nt = int(off[-1]), len(lens)
    cams = np.zeros((num_images, 18))
    cams[:, [0, 4, 8]] = 1.0
    cams[:, 9:12] = rng.normal(size=(num_images, 3))
    fo = 4 * np.arange(num_images + 1, dtype=np.int64)
    return {"cameras": cams, "reconstructed": (rng.random(num_images) < 0.7).astype(np.uint8),
            "intrinsic_group": rng.integers(0, 3, num_images).astype(np.uint32),
            "group_intrinsics": rng.normal(size=(3, 6)), "feature_offsets": fo,
            "features": rng.normal(size=(4 * num_images, 2)).astype(np.float32), "points": rng.normal(size=(nt, 3)),
            "track_offsets": off, "track_image": rng.integers(0, num_images, ne).astype(np.uint32),
            "track_feature": rng.integers(0, 4, ne).astype(np.uint32)}


LENS = {
    "one": [1], "tile": [2] * 1024, "tile + 1": [2] * 1024 + [1], "tile - 1": [1] * 2047,
    "empty runs": [0] * 5 + [2047] + [0] * 3000 + [1] + [0] * 7 + [1, 0, 0, 5] + [0] * 4,
    "long": [3, 7000, 2], "many": list(np.random.default_rng(1).integers(0, 9, 5000)),
}


@pytest.mark.parametrize("lens", sorted(LENS))
@pytest.mark.parametrize("images", [1, 127, 128, 129, 8192, 8193, 20000])
def test_pack_matches_numpy(lens, images, handle, abi):
    s = state(LENS[lens], images, seed=images)
    pk = abi.EnginePack(s)
    st, o = pk.pack(handle.lib, handle.h, -1, abi.LOCK_NONE)
    handle.check(st, "gbsfm_pack_ba")
    r = pk.result(o)
    rec = s["reconstructed"].astype(bool)
    img, off = s["track_image"], s["track_offsets"]
    keep = rec[img]
    ordinal = np.cumsum(rec) - 1
    assert o.num_cameras == rec.sum() and o.num_observations == keep.sum()
    np.testing.assert_array_equal(r["camera_image"], np.flatnonzero(rec))
    np.testing.assert_array_equal(r["camera_index"], ordinal[img[keep]])
    np.testing.assert_array_equal(r["intrinsic_index"], s["intrinsic_group"][img[keep]])
    np.testing.assert_array_equal(r["point_index"], np.repeat(np.arange(len(off) - 1), np.diff(off))[keep])
    np.testing.assert_array_equal(r["observations"],
                                  s["features"][4 * img[keep].astype(np.int64) + s["track_feature"][keep]].astype(float))
    np.testing.assert_array_equal(r["extrinsics"][:, 3:], s["cameras"][rec, 9:12])

"""FP32 triangulation: the batch sizes where the launch changes its block size
and the camera counts on both sides of the shared-memory table.  A track's
result does not depend on its neighbours or its block, so a batch's results
equal, bit for bit, those of its tracks given in reverse order and of a part
of them in a smaller batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def triangulate(handle, abi, tr, pick):
    off = tr["track_offsets"]
    lens = (off[1:] - off[:-1])[pick]
    idx = np.concatenate([np.arange(off[t], off[t + 1]) for t in pick])
    offs = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint32)
    cam = np.ascontiguousarray(tr["camera_index"][idx])
    xy = np.ascontiguousarray(tr["xy"][idx], dtype=np.float32)
    P = np.ascontiguousarray(tr["P"], dtype=np.float32)
    n = len(pick)
    X, st, md = np.zeros((n, 3), np.float32), np.zeros(n, np.uint8), np.zeros(n, np.float32)
    rc = handle.lib.gbtri_nview_batched_f32(handle.h, abi.TRI_NVIEW, P.ctypes.data, len(P), offs.ctypes.data,
                                            cam.ctypes.data, xy.ctypes.data, n, 1, X.ctypes.data, st.ctypes.data,
                                            md.ctypes.data, abi.MEMORY_HOST)
    handle.check(rc, "gbtri_nview_batched_f32")
    return X, st, md


@pytest.mark.parametrize("tracks,cameras", [(1, 20), (63, 20), (65, 20), (77824, 40), (311296, 40), (311297, 40),
                                            (400, 1024), (400, 1025), (80000, 1024)])
def test_results_do_not_depend_on_the_batch(tracks, cameras, handle, abi, scenes):
    tr = scenes.track_scene(num_cameras=cameras, num_tracks=tracks, seed=21, min_len=2, max_len=8)
    every = np.arange(tracks)
    a = triangulate(handle, abi, tr, every)
    part = every[::max(1, tracks // 200)]
    b = triangulate(handle, abi, tr, part[::-1].copy())
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x[part], y[::-1])

"""The gradient's fixed-point scale comes from the largest term of each entry.
Points with one observation each, seen by a camera at the origin with f = 1:
the Jacobian is (1, 0, -x; 0, 1, -y) and the residual a difference of two
doubles, so an entry's one term t is known to a few roundings.  With n
observations the scale 2^k has t n < 2^(62 - k) for the smallest such power, and
the entry is off by half a unit, 2^(-k - 1), beside the roundings: 4 of 2^-53 of
the products' size."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("stored", [False, True])
@pytest.mark.parametrize("n", [1 << 16, 70001])
def test_single_terms_keep_the_bits_of_their_scale(n, stored, mixed, handle, abi):
    rng = np.random.default_rng(n)
    xy = rng.uniform(0.5, 1.0, (n, 2))
    sc = dict(model=0, extrinsics=np.zeros((1, 6)), intrinsics=np.ones((1, 1)),
              points=np.concatenate([xy, np.ones((n, 1))], 1), observations=rng.uniform(-1, 1, (n, 2)),
              camera_index=np.zeros(n, np.uint32), intrinsic_index=np.zeros(n, np.uint32),
              point_index=np.arange(n, dtype=np.uint32))
    p = (hp := abi.HostProblem(sc)).struct()
    g = np.zeros(7 + 3 * n)
    blocks = [np.zeros((n, w)) for w in (12, 2, 6)] if stored else [None] * 3
    fn = handle.lib.gbba_project_backward_mixed if mixed else handle.lib.gbba_project_backward
    handle.check(fn(handle.h, C.byref(p), abi.LOSS_SQUARED, 1.0,
                    *[b.ctypes.data if b is not None else None for b in blocks], g.ctypes.data), "backward")
    r = xy - hp.observations.reshape(n, 2)
    z = -(xy.astype(np.float32) if mixed else xy).astype(np.longdouble)
    t = np.concatenate([r, ((z * r).sum(1))[:, None]], 1)
    size = np.concatenate([np.abs(r), np.abs(z * r).sum(1)[:, None]], 1)
    e = np.frexp(np.abs(t).astype(np.float64) * n)[1]
    bound = np.ldexp(0.5, e - 62) + 4 * 2.0**-53 * size
    assert (np.abs(g[7:].reshape(n, 3) - t) <= bound).all()

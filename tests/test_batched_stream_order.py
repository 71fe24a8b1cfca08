"""A batch in device memory whose arrays are still being written by work on the
default stream when the call is made: the call comes after that work, whatever
stream it runs on, so the solve is the same bit for bit as one whose arrays
were complete."""
import ctypes as C

import numpy as np
import pytest

from test_ba_gpu import local_problems

pytestmark = pytest.mark.gpu

ARRAYS = ("extrinsics", "intrinsics", "points", "observations", "camera_index", "intrinsic_index", "point_index")


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("own_stream", [True, False])
def test_arrays_from_the_default_stream(own_stream, precision, handle, abi, scenes):
    import torch
    o = abi.default_options(precision=abi.PRECISION_MIXED if precision == "mixed" else abi.PRECISION_FP64,
                            max_num_iterations=3)
    other = torch.cuda.Stream()
    if not own_stream:
        o.stream = other.cuda_stream
    probs = local_problems(scenes, 3, seed=931)
    runs = []
    for late in (False, True):
        dev = [abi.DeviceProblem(p) for p in probs]
        good = [{f: getattr(d, f).clone() for f in ARRAYS} for d in dev]
        if late:
            for d in dev:
                for f in ARRAYS:
                    getattr(d, f).zero_()  # (valid indices)
        torch.cuda.synchronize()
        if late:
            torch.cuda._sleep(200_000_000)  # about 0.1 s in front of the copies
            for d, g in zip(dev, good):
                for f in ARRAYS:
                    getattr(d, f).copy_(g[f])
        structs = (abi.GbbaProblem * 3)(*[d.struct() for d in dev])
        s = (abi.GbbaSummary * 3)()
        handle.check(handle.lib.gbba_solve_batched(handle.h, structs, 3, C.byref(o), s), "batched")
        runs.append(([x.final_cost for x in s], [d.params() for d in dev]))
    assert runs[0][0] == runs[1][0] and min(runs[0][0]) > 0
    for a, b in zip(runs[0][1], runs[1][1]):
        for f in a:
            np.testing.assert_array_equal(a[f], b[f])

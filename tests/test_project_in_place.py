"""The projection's arrays in device memory: used where they are when the kernels
can, copied otherwise.  Arrays off their type's alignment, outputs over inputs
and outputs over each other give what separate, aligned arrays give (of
outputs over each other the last in the order of the arguments stays)."""
import ctypes as C

import numpy as np
import pytest

from test_camera_lin import scene

pytestmark = pytest.mark.gpu

ARRAYS = ("extrinsics", "intrinsics", "points", "observations", "camera_index", "intrinsic_index", "point_index")


class Buffer:
    """Device bytes; put() returns the address of a copy at an odd place."""

    def __init__(self, size):
        import torch
        self.torch, self.b, self.used = torch, torch.zeros(size, dtype=torch.uint8, device="cuda:0"), 0

    def place(self, nbytes, off):
        at = (self.used + 255) // 256 * 256 + off
        self.used = at + nbytes
        assert self.used <= self.b.numel()
        return at

    def put(self, a, off):
        raw = np.ascontiguousarray(a).view(np.uint8).reshape(-1)
        at = self.place(raw.size, off)
        self.b[at:at + raw.size] = self.torch.from_numpy(raw.copy()).to("cuda:0")
        return self.b.data_ptr() + at

    def get(self, at, count):
        return self.b[at:at + 8 * count].cpu().numpy().copy().view(np.float64)


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("model", [0, 1, 2])
@pytest.mark.parametrize("kind", ["aligned", "odd", "over inputs", "over outputs"])
def test_any_place_gives_the_same(kind, model, mixed, handle, abi, scenes):
    import torch
    sc = scene(scenes, abi, model)
    hp = abi.HostProblem(sc)
    p, k = hp.struct(), abi.MODEL_K[model]
    no, ng = p.num_observations, 6 * p.num_cameras + k * p.num_intrinsics + 3 * p.num_points
    fn = handle.lib.gbba_project_backward_mixed if mixed else handle.lib.gbba_project_backward
    counts = [12 * no, 2 * k * no, 6 * no, ng, 2 * no]  # the backward outputs, then the residuals
    ref = [np.zeros(c) for c in counts]
    cost = C.c_double()
    handle.check(fn(handle.h, C.byref(p), 1, 4.0, *[r.ctypes.data for r in ref[:4]]), "backward")
    handle.check(handle.lib.gbba_project_forward(handle.h, C.byref(p), 1, 4.0, ref[4].ctypes.data, C.byref(cost)),
                 "forward")
    want = cost.value

    buf = Buffer(1 << 20)
    p.memory = abi.MEMORY_DEVICE
    odd = kind == "odd"
    at = {}
    for f in ARRAYS:
        off = (2 if f.endswith("index") else 4) if odd else 0
        setattr(p, f, buf.put(getattr(hp, f), off))
        at[f] = getattr(p, f) - buf.b.data_ptr()
    outs = [buf.place(8 * c, 4 if odd else 0) for c in counts]
    if kind == "over inputs":
        outs[4] = at["observations"]          # residuals over the observations
        outs[3] = at["extrinsics"]            # gradient over the parameters and what follows
        buf.place(8 * ng, 0)
    if kind == "over outputs":
        outs[2] = outs[0]                     # jac_point and the extrinsic blocks
        outs[1] = outs[0] + 8 * 6 * no
    torch.cuda.synchronize()
    base = buf.b.data_ptr()
    handle.check(handle.lib.gbba_project_forward(handle.h, C.byref(p), 1, 4.0, base + outs[4], C.byref(cost)), "forward")
    np.testing.assert_array_equal(buf.get(outs[4], counts[4]), ref[4])
    assert cost.value == want
    if kind == "over inputs":  # the observations again
        buf.b[at["observations"]:][:16 * no] = torch.from_numpy(hp.observations.view(np.uint8).reshape(-1).copy()).to("cuda:0")
        torch.cuda.synchronize()
    handle.check(fn(handle.h, C.byref(p), 1, 4.0, *[base + o for o in outs[:4]]), "backward")
    for i in ((3,) if kind == "over outputs" else (0, 1, 2, 3)):
        np.testing.assert_array_equal(buf.get(outs[i], counts[i]), ref[i])
    if kind == "over outputs":
        np.testing.assert_array_equal(buf.get(outs[2], counts[2]), ref[2])
        tail = buf.get(outs[1], counts[1])
        np.testing.assert_array_equal(tail, ref[1])

"""Performance cases: the calls that a reconstruction program makes into the
engine, through the C ABI, over the sizes that it meets.

Every case names an entry point (`kind`) and its sizes:

  solve      gbba_solve: two-view refinement, the incremental engine's bundle
             adjustment (intrinsic groups shared by its cameras), the global
             one (intrinsics per camera) on the dense and the iterative path
  windows    gbba_solve_batched: local windows, one call
  backward   gbba_project_backward: residual Jacobians and the gradient
  tri_f32    gbtri_nview_batched_f32: all tracks, N-view + one Gauss-Newton step
  tri_f64    gbtri_nview_batched: the same estimator in FP64
  pack       gbsfm_pack_ba: the engine's maps to a bundle-adjustment problem
  acransac   gbsfm_acransac_score: candidate models of a robust resection

Inputs are seeded synthetic scenes with the distributions of the package's
scene generators, drawn on the GPU.  A program keeps one handle, and so does
this file.
"""
import ctypes as C
import importlib
import math

import numpy as np
import torch

_gb = importlib.import_module("3dreconstruction_gb300")
abi = importlib.import_module("3dreconstruction_gb300.abi")

DEV = "cuda:0"
F64 = torch.float64
PP = (960.0, 540.0)
_kept = {}


def _handle():
    if "handle" not in _kept:
        _kept["handle"] = _gb.Handle(0)
    return _kept["handle"]


def _stream():
    if "stream" not in _kept:
        _kept["stream"] = torch.cuda.Stream(DEV)
    return _kept["stream"]


# --------------------------------------------------------------------- cases
def listed():
    return [
        # The refinement after a relative pose: two cameras, a few hundred
        # matches, host arrays.  The smallest solve; hundreds of them run at
        # the start of a global reconstruction.
        dict(name="solve two views", kind="solve", cameras=2, points=400, views=2, model="pinhole", intrinsics="held",
             precision="fp64", solver="auto", iterations=20, hold=1, local=False, memory="host"),
        # The incremental engine's bundle adjustment after a handful of
        # images: one camera body, so one intrinsic group for all; host arrays.
        dict(name="solve window shared", kind="solve", cameras=20, points=2000, views=5, model="k3",
             intrinsics="1 groups", precision="fp64", solver="auto", iterations=10, hold=2, local=True, memory="host"),
        # The same engine late in a reconstruction: three camera bodies, the
        # map resident on the device.
        dict(name="solve map shared", kind="solve", cameras=300, points=60000, views=10, model="k3",
             intrinsics="3 groups", precision="fp64", solver="auto", iterations=5, hold=2, local=True,
             memory="device"),
        # A global bundle adjustment of unordered photographs, intrinsics per
        # camera, default precision.
        dict(name="solve global fp64", kind="solve", cameras=200, points=40000, views=10, model="k3",
             intrinsics="own", precision="fp64", solver="auto", iterations=5, hold=2, local=False, memory="device"),
        # The benchmark's medium workload: dense Schur in mixed precision.
        dict(name="solve medium mixed", kind="solve", cameras=500, points=200000, views=10, model="k3",
             intrinsics="own", precision="mixed", solver="auto", iterations=10, hold=2, local=False, memory="device"),
        # The benchmark's large workload: 20M observations on the iterative path.
        dict(name="solve large pcg", kind="solve", cameras=5000, points=2000000, views=10, model="k3",
             intrinsics="own", precision="mixed", solver="auto", iterations=4, hold=2, local=False, memory="device"),
        # Local windows of a long sequence, two for each multiprocessor.
        dict(name="windows mixed", kind="windows", windows=304, min_cameras=5, max_cameras=40, min_points=200,
             max_points=5000, precision="mixed", iterations=6),
        # Jacobians and gradient for a caller's own optimiser.
        dict(name="backward 1M", kind="backward", cameras=300, points=100000, views=10, precision="fp64"),
        # The benchmark's triangulation workload.
        dict(name="tri f32 1M", kind="tri_f32", cameras=200, tracks=1000000, min_len=2, max_len=30, steps=1),
        # The FP64 estimator over the tracks of a middle-sized map.
        dict(name="tri f64 100k", kind="tri_f64", cameras=200, tracks=100000, min_len=2, max_len=30),
        # The engine's maps of the large workload into a problem.
        dict(name="pack 10M", kind="pack", images=5000, points=2000000, max_len=8),
        # Candidate models of one robust resection.
        dict(name="acransac 1024", kind="acransac", models=1024, points=2000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["two views", "shared", "global fp64", "mixed", "pcg", "windows", "backward", "tri_f32",
                       "tri_f64", "pack", "acransac"])
    if what == "two views":
        return dict(kind="solve", cameras=2, points=_log(rng, 50, 4000), views=2, model="pinhole", intrinsics="held",
                    precision="fp64", solver="auto", iterations=20, hold=1, local=False, memory="host")
    if what == "shared":
        nc = _log(rng, 5, 300)
        return dict(kind="solve", cameras=nc, points=nc * _log(rng, 50, 200), views=min(nc, rng.randint(3, 10)),
                    model=rng.choice(["k3", "t2"]), intrinsics="%d groups" % rng.randint(1, min(4, nc)),
                    precision="fp64", solver="auto", iterations=rng.randint(3, 6), hold=2, local=True,
                    memory=rng.choice(["host", "device"]))
    if what == "global fp64":
        nc = _log(rng, 10, 200)
        return dict(kind="solve", cameras=nc, points=nc * _log(rng, 50, 200), views=min(nc, rng.randint(4, 10)),
                    model=rng.choice(["k3", "t2"]), intrinsics="own", precision="fp64", solver="auto",
                    iterations=rng.randint(3, 6), hold=2, local=False, memory="device")
    if what == "mixed":
        nc = _log(rng, 50, 500)
        return dict(kind="solve", cameras=nc, points=nc * _log(rng, 100, 400), views=rng.randint(5, 10), model="k3",
                    intrinsics="own", precision="mixed", solver="auto", iterations=rng.randint(3, 8), hold=2,
                    local=rng.random() < 0.5, memory="device")
    if what == "pcg":
        nc = _log(rng, 1500, 5000)
        return dict(kind="solve", cameras=nc, points=nc * _log(rng, 50, 400), views=rng.randint(5, 10), model="k3",
                    intrinsics="own", precision="mixed", solver="iterative", iterations=rng.randint(2, 4), hold=2,
                    local=False, memory="device")
    if what == "windows":
        lo = rng.randint(5, 12)
        return dict(kind="windows", windows=_log(rng, 20, 304), min_cameras=lo, max_cameras=rng.randint(lo, 40),
                    min_points=200, max_points=_log(rng, 300, 5000), precision="mixed", iterations=rng.randint(3, 6))
    if what == "backward":
        return dict(kind="backward", cameras=_log(rng, 5, 300), points=_log(rng, 500, 100000),
                    views=rng.randint(3, 10), precision=rng.choice(["fp64", "fp64", "mixed"]))
    if what in ("tri_f32", "tri_f64"):
        top = 1000000 if what == "tri_f32" else 100000
        lo = rng.randint(2, 5)
        d = dict(kind=what, cameras=_log(rng, 20, 900), tracks=_log(rng, 500, top), min_len=lo,
                 max_len=rng.randint(lo, 20))
        return dict(d, steps=rng.randint(0, 2)) if what == "tri_f32" else d
    if what == "pack":
        return dict(kind="pack", images=_log(rng, 60, 5000), points=_log(rng, 1000, 2000000),
                    max_len=rng.randint(3, 8))
    return dict(kind="acransac", models=_log(rng, 16, 1024), points=_log(rng, 30, 4000))


# -------------------------------------------------------------------- scenes
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 2654435761 % (1 << 62) + 17)
    return g


def _sizes(g, draw, n):
    """n sizes from draw(generator): the same ones for every seed, in the
    seed's order, so that a case has one shape."""
    fixed = torch.Generator(device=DEV)
    fixed.manual_seed(20260 + n)
    return draw(fixed)[torch.randperm(n, generator=g, device=DEV)]


def _u(g, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(*shape, generator=g, device=DEV, dtype=F64)


def _n(g, sigma, *shape):
    return sigma * torch.randn(*shape, generator=g, device=DEV, dtype=F64)


def _ints(g, lo, hi, *shape):  # lo..hi, both included
    return torch.randint(lo, hi + 1, shape, generator=g, device=DEV)


def _look_at(centers):
    """Rotations whose z axis points from the centres to the origin."""
    z = -centers / centers.norm(dim=-1, keepdim=True)
    up = torch.tensor([0.0, 1.0, 0.0], device=DEV, dtype=F64).expand_as(z)
    x = torch.linalg.cross(up, z)
    x = x / x.norm(dim=-1, keepdim=True)
    return torch.stack([x, torch.linalg.cross(z, x), z], -2)


def _rotation(w):
    """Rotation matrices of angle-axis vectors."""
    th = w.norm(dim=-1).clamp_min(1e-300)
    k = w / th[..., None]
    K = torch.zeros(w.shape[:-1] + (3, 3), device=DEV, dtype=F64)
    K[..., 0, 1], K[..., 0, 2], K[..., 1, 2] = -k[..., 2], k[..., 1], -k[..., 0]
    K[..., 1, 0], K[..., 2, 0], K[..., 2, 1] = k[..., 2], -k[..., 1], k[..., 0]
    s, c = torch.sin(th)[..., None, None], torch.cos(th)[..., None, None]
    return torch.eye(3, device=DEV, dtype=F64) + s * K + (1 - c) * (K @ K)


def _angle_axis(R):
    """Angle-axis vectors of rotations away from half turns."""
    cos = ((R.diagonal(dim1=-2, dim2=-1).sum(-1) - 1) / 2).clamp(-1, 1)
    th = torch.acos(cos)
    w = torch.stack([R[..., 2, 1] - R[..., 1, 2], R[..., 0, 2] - R[..., 2, 0], R[..., 1, 0] - R[..., 0, 1]], -1)
    s = torch.sin(th)
    return w * torch.where(s < 1e-9, torch.full_like(th, 0.5), th / (2 * s.clamp_min(1e-9)))[..., None]


def _sphere(g, n, radius):
    i = torch.arange(n, device=DEV, dtype=F64) + 0.5
    y = math.sin(math.radians(60)) * (1 - 2 * i / n)
    phi = i * math.pi * (3 - math.sqrt(5.0)) + _u(g, 0, 2 * math.pi, 1)
    r = (1 - y * y).sqrt()
    return radius * torch.stack([r * torch.cos(phi), y, r * torch.sin(phi)], -1)


def _arc(g, n, radius, span):
    a = torch.linspace(-span, span, n, device=DEV, dtype=F64) + _u(g, -0.3, 0.3, n) * span / n
    return radius * torch.stack([torch.sin(a), _u(g, -0.02, 0.02, n), torch.cos(a)], -1)


def _distort(model, k, x, y):
    """Predicted pixels (model 0: f; 1: radial K3; 2: Brown-T2) of normalised points."""
    if model == 0:
        return k[:, 0] * x, k[:, 0] * y
    r2 = x * x + y * y
    rc = 1 + k[:, 3] * r2 + k[:, 4] * r2 * r2 + k[:, 5] * r2 * r2 * r2
    xd, yd = x * rc, y * rc
    if model == 2:
        xd, yd = (xd + 2 * k[:, 6] * x * y + k[:, 7] * (r2 + 2 * x * x),
                  yd + 2 * k[:, 7] * x * y + k[:, 6] * (r2 + 2 * y * y))
    return k[:, 1] + k[:, 0] * xd, k[:, 2] + k[:, 0] * yd


def _tracks(g, num, lens, num_cameras, local):
    """CSR tracks over distinct cameras, ascending inside a track: start +
    j step (mod the cameras), any step coprime to their number, or a step of 1
    to 4 that stays inside the sequence (local)."""
    lens = lens.clamp_max(num_cameras)
    tr = torch.repeat_interleave(torch.arange(num, device=DEV), lens)
    off = torch.zeros(num + 1, dtype=torch.int64, device=DEV)
    off[1:] = torch.cumsum(lens, 0)
    j = torch.arange(len(tr), device=DEV) - off[tr]
    if local:
        last = (lens - 1).clamp_min(1)
        step = torch.minimum(_ints(g, 1, 4, num), ((num_cameras - 1) // last).clamp_min(1))
        start = (torch.rand(num, generator=g, device=DEV, dtype=F64) * (num_cameras - (lens - 1) * step)).long()
        cam = start[tr] + j * step[tr]
    else:
        steps = torch.tensor([s for s in range(1, max(2, num_cameras)) if math.gcd(s, num_cameras) == 1], device=DEV)
        start = _ints(g, 0, num_cameras - 1, num)
        step = steps[_ints(g, 0, len(steps) - 1, num)]
        cam = (start[tr] + j * step[tr]) % num_cameras
        order = torch.sort(tr * num_cameras + cam).indices
        cam = cam[order]
    return off, tr, cam


MODELS = {"pinhole": 0, "k3": 1, "t2": 2}


def _ba_scene(g, nc, npts, views, model, groups, local, sigma=0.6, outliers=0.03, rot=0.01, shift=0.05, xs=0.05,
              hold=2):
    """A perturbed bundle-adjustment scene as CUDA tensors.  groups: 0 = one
    intrinsic block per camera, n = n blocks shared round robin."""
    k = abi.MODEL_K[model]
    if local or nc < 4:
        centers, extent = _arc(g, nc, 10.0, min(2.6, 0.12 * nc)), 2.0
    else:
        centers, extent = _sphere(g, nc, 15.0), 3.0
    R = _look_at(centers)
    t = -(R @ centers[..., None])[..., 0]
    ext = torch.cat([_angle_axis(R), t], 1)
    ni = groups or nc
    intr = torch.zeros(ni, k, device=DEV, dtype=F64)
    intr[:, 0] = _u(g, 900, 1100, ni)
    if model:
        intr[:, 1], intr[:, 2] = PP
        for c, s in ((3, 0.05), (4, 0.01), (5, 0.01)):
            intr[:, c] = _n(g, s, ni)
    if model == 2:
        intr[:, 6:8] = _n(g, 0.002, ni, 2)
    X = _u(g, -extent, extent, npts, 3)
    lens = _sizes(g, lambda f: 2 + torch.poisson(torch.full((npts,), views - 2.0, device=DEV), generator=f).long(), npts)
    _, pt, cam = _tracks(g, npts, lens, nc, local)
    icam = cam % ni
    p = (_rotation(ext[:, :3])[cam] @ X[pt][..., None])[..., 0] + ext[cam, 3:]
    u, v = _distort(model, intr[icam], p[:, 0] / p[:, 2], p[:, 1] / p[:, 2])
    obs = torch.stack([u, v], 1) + _n(g, sigma, len(pt), 2)
    if outliers:
        bad = torch.rand(len(pt), generator=g, device=DEV) < outliers
        box = torch.stack([_u(g, 0, 1920, len(pt)), _u(g, 0, 1080, len(pt))], 1)
        if model == 0:
            box = box - torch.tensor(PP, device=DEV, dtype=F64)
        obs = torch.where(bad[:, None], box, obs)

    def unit(*shape):
        a = _n(g, 1.0, *shape)
        return a / a.norm(dim=-1, keepdim=True)

    held = torch.arange(nc, device=DEV) < hold
    step = torch.cat([rot * unit(nc, 3), shift * unit(nc, 3)], 1)
    ext = ext + torch.where(held[:, None], torch.zeros_like(step), step)
    intr = intr.clone()
    intr[:, 0] *= 1 + _n(g, 0.002, ni)
    return dict(model=model, extrinsics=ext, intrinsics=intr, points=X + _n(g, xs, npts, 3), observations=obs,
                camera_index=cam.int(), intrinsic_index=icam.int(), point_index=pt.int(),
                camera_constant=held.to(torch.uint8))


class _Device:
    """A gbba_problem over CUDA tensors."""

    memory = abi.MEMORY_DEVICE

    def __init__(self, s):
        self.a = {f: s[f].contiguous() for f in abi.HostProblem.FIELDS if s.get(f) is not None}
        self.model = s["model"]

    def ptr(self, f):
        return self.a[f].data_ptr()

    def count(self, f):
        return self.a[f].numel()

    def struct(self):
        p = abi.GbbaProblem()
        p.camera_model, p.memory = self.model, self.memory
        p.num_cameras = self.count("extrinsics") // 6
        p.num_intrinsics = self.count("intrinsics") // abi.MODEL_K[self.model]
        p.num_points = self.count("points") // 3
        p.num_observations = self.count("observations") // 2
        for f in self.a:
            setattr(p, f, self.ptr(f))
        return p


class _Host(_Device):
    """The same over numpy arrays."""

    memory = abi.MEMORY_HOST

    def __init__(self, s):
        super().__init__(s)
        self.a = {f: v.cpu().numpy() for f, v in self.a.items()}

    def ptr(self, f):
        return self.a[f].ctypes.data

    def count(self, f):
        return self.a[f].size


PARAMS = ("extrinsics", "intrinsics", "points")


def _groups(case):
    return {"own": 0, "held": 1}.get(case["intrinsics"]) if case["intrinsics"] in ("own", "held") else \
        int(case["intrinsics"].split()[0])


def _scene_of(case, seed):
    s = _ba_scene(_gen(seed), case["cameras"], case["points"], case["views"], MODELS[case["model"]], _groups(case),
                  case["local"], hold=case["hold"])
    if case["intrinsics"] == "held":
        s["intrinsic_constant"] = torch.ones(len(s["intrinsics"]), dtype=torch.uint8, device=DEV)
    return s


# ------------------------------------------------------------------- prepare
def prepare(case, seed):
    state = globals()["_prepare_" + case["kind"]](case, seed)
    torch.cuda.synchronize()  # the handle works on a stream of its own
    return state


def run(state):
    return globals()["_run_" + state["kind"]](state)


def _prepare_solve(case, seed):
    s = _scene_of(case, seed)
    p = (_Host if case["memory"] == "host" else _Device)(s)
    o = abi.default_options(
        max_num_iterations=case["iterations"], loss_type=abi.LOSS_HUBER, loss_scale=4.0, fp64_polish_iterations=0,
        precision=abi.PRECISION_MIXED if case["precision"] == "mixed" else abi.PRECISION_FP64,
        linear_solver=abi.SOLVER_ITERATIVE_SCHUR if case["solver"] == "iterative" else abi.SOLVER_AUTO)
    o.stream = _stream().cuda_stream
    copy = np.copy if case["memory"] == "host" else torch.clone
    return dict(kind="solve", problem=p, struct=p.struct(), options=o, start={f: copy(p.a[f]) for f in PARAMS},
                handle=_handle())


def _run_solve(st):
    # the map as it stands before this bundle adjustment, refined in place
    a, h = st["problem"].a, st["handle"]
    if isinstance(a["points"], np.ndarray):
        for f in PARAMS:
            np.copyto(a[f], st["start"][f])
    else:
        with torch.cuda.stream(_stream()):
            for f in PARAMS:
                a[f].copy_(st["start"][f])
    s = abi.GbbaSummary()
    h.check(h.lib.gbba_solve(h.h, C.byref(st["struct"]), C.byref(st["options"]), C.byref(s)), "gbba_solve")
    return dict({f: a[f] for f in PARAMS}, initial_cost=s.initial_cost, final_cost=s.final_cost,
                iterations=s.num_iterations, successful=s.num_successful_steps, termination=s.termination_type)


def _prepare_windows(case, seed):
    g = _gen(seed)
    nw = case["windows"]
    size = _sizes(g, lambda f: torch.stack([_ints(f, case["min_cameras"], case["max_cameras"], nw),
                                            _ints(f, case["min_points"], case["max_points"], nw)], 1), nw)
    probs = []
    for c, n in size.tolist():
        centers = _arc(g, c, 8.0, 0.6)
        R = _look_at(centers)
        ext = torch.cat([_angle_axis(R), -(R @ centers[..., None])[..., 0]], 1)
        intr = torch.tensor([[1000.0, PP[0], PP[1], 0.02, -0.005, 0.004, 0.001, -0.002]], device=DEV, dtype=F64)
        X = _u(g, -2.0, 2.0, n, 3)
        _, pt, cam = _tracks(g, n, _sizes(g, lambda f: _ints(f, 2, c, n), n), c, False)
        p = (R[cam] @ X[pt][..., None])[..., 0] + ext[cam, 3:]
        u, v = _distort(2, intr.expand(len(pt), 8), p[:, 0] / p[:, 2], p[:, 1] / p[:, 2])
        held = torch.arange(c, device=DEV) < 2
        step = torch.cat([_n(g, 0.01, c, 3), _n(g, 0.03, c, 3)], 1)
        probs.append(_Host(dict(
            model=2, extrinsics=ext + torch.where(held[:, None], torch.zeros_like(step), step),
            intrinsics=intr * torch.tensor([1.001] + [1.0] * 7, device=DEV, dtype=F64), points=X + _n(g, 0.05, n, 3),
            observations=torch.stack([u, v], 1) + _n(g, 0.5, len(pt), 2), camera_index=cam.int(),
            intrinsic_index=torch.zeros_like(cam).int(), point_index=pt.int(),
            camera_constant=held.to(torch.uint8))))
    # the windows' parameters in three arrays, a window's block its slice
    now, start = {}, {}
    for f in PARAMS:
        now[f] = np.concatenate([p.a[f] for p in probs])
        start[f] = now[f].copy()
        at = np.cumsum([0] + [len(p.a[f]) for p in probs])
        for i, p in enumerate(probs):
            p.a[f] = now[f][at[i]:at[i + 1]]
    structs = (abi.GbbaProblem * nw)(*[p.struct() for p in probs])
    o = abi.default_options(max_num_iterations=case["iterations"], loss_type=abi.LOSS_HUBER, loss_scale=4.0,
                            fp64_polish_iterations=0,
                            precision=abi.PRECISION_MIXED if case["precision"] == "mixed" else abi.PRECISION_FP64)
    return dict(kind="windows", keep=probs, structs=structs, options=o, now=now, start=start, n=nw, handle=_handle())


def _run_windows(st):
    h = st["handle"]
    for f in PARAMS:
        np.copyto(st["now"][f], st["start"][f])
    sums = (abi.GbbaSummary * st["n"])()
    h.check(h.lib.gbba_solve_batched(h.h, st["structs"], st["n"], C.byref(st["options"]), sums), "gbba_solve_batched")
    return dict(st["now"], final_cost=np.array([s.final_cost for s in sums]),
                iterations=np.array([s.num_iterations for s in sums]),
                termination=np.array([s.termination_type for s in sums]))


def _prepare_backward(case, seed):
    p = _Device(_ba_scene(_gen(seed), case["cameras"], case["points"], case["views"], 1, 0, False))
    no, nc, npt = p.count("observations") // 2, p.count("extrinsics"), p.count("points")

    def out(*shape):
        return torch.zeros(*shape, dtype=F64, device=DEV)

    return dict(kind="backward", problem=p, struct=p.struct(), handle=_handle(), mixed=case["precision"] == "mixed",
                je=out(no, 2, 6), ji=out(no, 2, 6), jp=out(no, 2, 3), grad=out(nc + p.count("intrinsics") + npt))


def _run_backward(st):
    h = st["handle"]
    f = h.lib.gbba_project_backward_mixed if st["mixed"] else h.lib.gbba_project_backward
    h.check(f(h.h, C.byref(st["struct"]), abi.LOSS_HUBER, 4.0, st["je"].data_ptr(), st["ji"].data_ptr(),
              st["jp"].data_ptr(), st["grad"].data_ptr()), "gbba_project_backward")
    return {k: st[k] for k in ("je", "ji", "jp", "grad")}


def _track_scene(case, seed):
    g = _gen(seed)
    nc, nt = case["cameras"], case["tracks"]
    centers = _sphere(g, nc, 15.0)
    R = _look_at(centers)
    t = -(R @ centers[..., None])[..., 0]
    K = torch.zeros(nc, 3, 3, device=DEV, dtype=F64)
    K[:, 0, 0] = K[:, 1, 1] = _u(g, 800, 1200, nc)
    K[:, 0, 2], K[:, 1, 2] = PP
    K[:, 2, 2] = 1
    P = K @ torch.cat([R, t[..., None]], 2)
    X = _u(g, -3.0, 3.0, nt, 3)
    off, tr, cam = _tracks(g, nt, _sizes(g, lambda f: _ints(f, case["min_len"], case["max_len"], nt), nt), nc, False)
    hom = (P[cam] @ torch.cat([X, torch.ones_like(X[:, :1])], 1)[tr][..., None])[..., 0]
    xy = hom[:, :2] / hom[:, 2:] + _n(g, 1.0, len(tr), 2)
    return P, off, tr, cam, xy


def _prepare_tri_f32(case, seed):
    P, off, _, cam, xy = _track_scene(case, seed)
    nt = case["tracks"]
    return dict(kind="tri_f32", handle=_handle(), P=P.float().contiguous(), off=off.int(), cam=cam.int(),
                xy=xy.float().contiguous(), nc=case["cameras"], nt=nt, steps=case["steps"],
                X=torch.zeros(nt, 3, device=DEV), status=torch.zeros(nt, dtype=torch.uint8, device=DEV),
                depth=torch.zeros(nt, device=DEV))


def _run_tri_f32(st):
    h = st["handle"]
    h.check(h.lib.gbtri_nview_batched_f32(
        h.h, abi.TRI_NVIEW, st["P"].data_ptr(), st["nc"], st["off"].data_ptr(), st["cam"].data_ptr(),
        st["xy"].data_ptr(), st["nt"], st["steps"], st["X"].data_ptr(), st["status"].data_ptr(),
        st["depth"].data_ptr(), abi.MEMORY_DEVICE), "gbtri_nview_batched_f32")
    return {k: st[k] for k in ("X", "status", "depth")}


def _prepare_tri_f64(case, seed):
    P, off, _, cam, xy = _track_scene(case, seed)
    return dict(kind="tri_f64", handle=_handle(), P=P.contiguous(), off=off, cam=cam.int(), xy=xy.contiguous(),
                nc=case["cameras"], nt=case["tracks"], X=torch.zeros(case["tracks"], 4, dtype=F64, device=DEV))


def _run_tri_f64(st):
    h = st["handle"]
    h.check(h.lib.gbtri_nview_batched(
        h.h, abi.TRI_NVIEW, st["P"].data_ptr(), st["nc"], st["off"].data_ptr(), st["cam"].data_ptr(),
        st["xy"].data_ptr(), st["nt"], st["X"].data_ptr(), None, abi.MEMORY_DEVICE), "gbtri_nview_batched")
    return st["X"]


def _pack_scene(case, seed):
    g = _gen(seed)
    ni, nt = case["images"], case["points"]
    centers = _sphere(g, ni, 12.0)
    R = _look_at(centers)
    cams = torch.cat([R.reshape(ni, 9), -(R @ centers[..., None])[..., 0], _u(g, 900, 1100, ni, 1),
                      torch.tensor([PP], device=DEV, dtype=F64).expand(ni, 2), _n(g, 0.02, ni, 3)], 1).contiguous()
    rec = (torch.rand(ni, generator=g, device=DEV) < 0.8).to(torch.uint8)
    nf = _ints(g, 20, 400, ni)
    fo = torch.zeros(ni + 1, dtype=torch.int64, device=DEV)
    fo[1:] = torch.cumsum(nf, 0)
    lens = _sizes(g, lambda f: _ints(f, 2, case["max_len"], nt), nt)
    off = torch.zeros(nt + 1, dtype=torch.int64, device=DEV)
    off[1:] = torch.cumsum(lens, 0)
    tr = torch.repeat_interleave(torch.arange(nt, device=DEV), lens)
    ne = len(tr)
    step = _ints(g, 1, 4, ne)
    step[off[:-1]] = 0
    cs = torch.cumsum(step, 0)
    start = _ints(g, 0, max(0, ni - 33), nt)
    img = (start[tr] + cs - cs[off[:-1]][tr]).clamp_max(ni - 1)
    return dict(cameras=cams, reconstructed=rec, intrinsic_group=_ints(g, 0, 2, ni).int(),
                group_intrinsics=_u(g, 900, 1100, 3, 6), feature_offsets=fo,
                features=_u(g, 0, 2000, int(fo[-1]), 2).float().contiguous(), points=_u(g, -2, 2, nt, 3),
                track_offsets=off, track_image=img.int(),
                track_feature=(torch.rand(ne, generator=g, device=DEV, dtype=F64) * nf[img]).int())


def _prepare_pack(case, seed):
    a = _pack_scene(case, seed)
    ni, nt, ne, nf = case["images"], case["points"], len(a["track_image"]), len(a["features"])
    s = abi.GbsfmEngineState()
    s.num_images, s.num_intrinsic_groups, s.num_features, s.num_points, s.num_entries = ni, 3, nf, nt, ne
    for k, v in a.items():
        setattr(s, k, v.data_ptr())
    out = dict(extrinsics=torch.zeros(ni, 6, dtype=F64, device=DEV), intrinsics=torch.zeros(3, 6, dtype=F64, device=DEV),
               points=torch.zeros(nt, 3, dtype=F64, device=DEV),
               observations=torch.zeros(ne, 2, dtype=F64, device=DEV),
               camera_constant=torch.zeros(ni, dtype=torch.uint8, device=DEV))
    for k, n in (("camera_index", ne), ("intrinsic_index", ne), ("point_index", ne), ("camera_image", ni)):
        out[k] = torch.zeros(n, dtype=torch.int32, device=DEV)
    o = abi.GbsfmBaArrays()
    for k, v in out.items():
        setattr(o, k, v.data_ptr())
    return dict(kind="pack", handle=_handle(), keep=a, state=s, arrays=o, out=out)


def _run_pack(st):
    h, o = st["handle"], st["arrays"]
    h.check(h.lib.gbsfm_pack_ba(h.h, C.byref(st["state"]), 7, abi.LOCK_AS_REFERENCE, C.byref(o), abi.MEMORY_DEVICE),
            "gbsfm_pack_ba")
    return dict(st["out"], counts=np.array([o.num_cameras, o.num_observations, o.measurements, o.locked_camera]))


def _resection(case, seed):
    g = _gen(seed)
    n, m = case["points"], case["models"]
    R = _look_at(torch.tensor([[0.5, -0.3, -8.0]], device=DEV, dtype=F64))[0]
    t = -(R @ torch.tensor([0.5, -0.3, -8.0], device=DEV, dtype=F64))
    X = _u(g, -2.5, 2.5, n, 3)
    p = X @ R.T + t
    x = p[:, :2] / p[:, 2:] + _n(g, 0.0005, n, 2)
    bad = torch.rand(n, generator=g, device=DEV) < 0.3
    x = torch.where(bad[:, None], _u(g, -0.9, 0.9, n, 2), x)
    # models of minimal samples: a third near the pose, the others off by more
    size = torch.where(torch.arange(m, device=DEV) % 3 == 0, 0.002, 0.05).to(F64)[:, None]
    Rm = _rotation(size * _n(g, 1.0, m, 3)) @ R
    return x.contiguous(), X, torch.cat([Rm, (t + size * 4 * _n(g, 1.0, m, 3))[..., None]], 2).reshape(m, 12)


def _prepare_acransac(case, seed):
    x, X, models = _resection(case, seed)
    n, m = case["points"], case["models"]
    return dict(kind="acransac", handle=_handle(), x=x, X=X.contiguous(), models=models.contiguous(), n=n, m=m,
                params=abi.GbsfmAcransacParams(6, 1, math.log10(math.pi), 1.0, math.inf),
                nfa=torch.zeros(m, dtype=F64, device=DEV), error_max=torch.zeros(m, dtype=F64, device=DEV),
                inliers=torch.zeros(m, dtype=torch.int32, device=DEV),
                order=torch.zeros(m, n, dtype=torch.int32, device=DEV))


def _run_acransac(st):
    h = st["handle"]
    h.check(h.lib.gbsfm_acransac_score(
        h.h, C.byref(st["params"]), st["n"], st["x"].data_ptr(), st["X"].data_ptr(), st["m"],
        st["models"].data_ptr(), st["nfa"].data_ptr(), st["inliers"].data_ptr(), st["error_max"].data_ptr(),
        st["order"].data_ptr(), abi.MEMORY_DEVICE), "gbsfm_acransac_score")
    return {k: st[k] for k in ("nfa", "error_max", "inliers", "order")}


# ---------------------------------------------------------------------- work
def _pairs(views):
    """Ordered observation pairs of a point: 2 + Poisson(views - 2) observations, half of n (n + 1)."""
    v = max(2.0, float(views))
    return 0.5 * (v * v + (v - 2.0) + v)


def work(case):
    kind = case["kind"]
    if kind == "solve":
        k = abi.MODEL_K[MODELS[case["model"]]]
        no, npts, nc = case["points"] * case["views"], case["points"], case["cameras"]
        free_i = 0 if case["intrinsics"] == "held" else k * (_groups(case) or nc)
        n = 6 * (nc - case["hold"]) + free_i
        b = 6 + k
        # per iteration and observation: residual, Jacobian, normal equations, back substitution
        flops = no * (250.0 + 12 * b + 4 * b * b)
        io = no * 28.0 + 2 * 8 * (6 * nc + (free_i or k) + 3 * npts)
        if case["solver"] == "auto" and n <= 16384:
            flops += npts * _pairs(case["views"]) * 6.0 * b * b + n ** 3 / 3.0
        return dict(bytes=io, flops=flops * case["iterations"])
    if kind == "windows":
        c = 0.5 * (case["min_cameras"] + case["max_cameras"])
        p = 0.5 * (case["min_points"] + case["max_points"])
        v = 0.5 * (2 + c)
        no = case["windows"] * p * v
        flops = no * (250.0 + 12 * 14 + 4 * 196) + case["windows"] * (p * 0.5 * v * (v + 1) * 216.0 + (6 * c + 8) ** 3 / 3)
        return dict(bytes=no * 28.0 + case["windows"] * 16.0 * (6 * c + 8 + 3 * p), flops=flops * case["iterations"])
    if kind == "backward":
        no = case["points"] * max(2, case["views"])
        n = 12 * case["cameras"] + 3 * case["points"]
        return dict(bytes=no * (28.0 + 8 * 30) + 16.0 * n, flops=no * 350.0)
    if kind in ("tri_f32", "tri_f64"):
        no = case["tracks"] * 0.5 * (case["min_len"] + case["max_len"])
        if kind == "tri_f32":
            return dict(bytes=12 * no + 21.0 * case["tracks"], flops=no * (200.0 + 90 * case["steps"]))
        return dict(bytes=20 * no + 40.0 * case["tracks"], flops=no * 200.0)
    if kind == "pack":
        ne = case["points"] * 0.5 * (2 + case["max_len"])
        return dict(bytes=8 * ne + 28 * 0.8 * ne + 56.0 * case["points"] + 200.0 * case["images"], flops=0)
    m, n = case["models"], case["points"]
    return dict(bytes=40.0 * n + m * (96 + 20 + 4.0 * n), flops=m * n * (30.0 + 2 * math.log2(n + 1)))


# --------------------------------------------------------------------- exact
def exact(case, seed):
    f = globals().get("_exact_" + case["kind"])
    return f(case, seed) if f else None


def _skew(v):
    z = torch.zeros_like(v[:, 0])
    return torch.stack([z, -v[:, 2], v[:, 1], v[:, 2], z, -v[:, 0], -v[:, 1], v[:, 0], z], 1).reshape(-1, 3, 3)


def _exact_backward(case, seed):
    """Jacobian blocks and gradient of the Huber-robustified residuals."""
    s = _ba_scene(_gen(seed), case["cameras"], case["points"], case["views"], 1, 0, False)
    c, gi, pt = s["camera_index"].long(), s["intrinsic_index"].long(), s["point_index"].long()
    w, X, k = s["extrinsics"][c, :3], s["points"][pt], s["intrinsics"][gi]
    R = _rotation(w)
    p = (R @ X[..., None])[..., 0] + s["extrinsics"][c, 3:]
    x, y, iz = p[:, 0] / p[:, 2], p[:, 1] / p[:, 2], 1 / p[:, 2]
    f = k[:, 0]
    r2 = x * x + y * y
    rc = 1 + k[:, 3] * r2 + k[:, 4] * r2 ** 2 + k[:, 5] * r2 ** 3
    dr = k[:, 3] + 2 * k[:, 4] * r2 + 3 * k[:, 5] * r2 ** 2
    r = torch.stack([k[:, 1] + f * x * rc, k[:, 2] + f * y * rc], 1) - s["observations"]
    A = f[:, None, None] * torch.stack([rc + 2 * x * x * dr, 2 * x * y * dr, 2 * x * y * dr, rc + 2 * y * y * dr],
                                       1).reshape(-1, 2, 2)
    z = torch.zeros_like(x)
    D = A @ torch.stack([iz, z, -x * iz, z, iz, -y * iz], 1).reshape(-1, 2, 3)
    th2 = (w * w).sum(1)
    th = th2.sqrt()
    W = _skew(w)
    Jr = torch.eye(3, device=DEV, dtype=F64) - ((1 - torch.cos(th)) / th2)[:, None, None] * W + \
        ((th - torch.sin(th)) / (th2 * th))[:, None, None] * (W @ W)
    je = torch.cat([D @ (-R @ _skew(X) @ Jr), D], 2)
    one = torch.ones_like(x)
    ji = torch.stack([x * rc, one, z, f * x * r2, f * x * r2 ** 2, f * x * r2 ** 3,
                      y * rc, z, one, f * y * r2, f * y * r2 ** 2, f * y * r2 ** 3], 1).reshape(-1, 2, 6)
    jp = D @ R
    sq = r.norm(dim=1)
    sr = torch.where(sq > 4.0, (4.0 / sq).sqrt(), torch.ones_like(sq))
    je, ji, jp, r = je * sr[:, None, None], ji * sr[:, None, None], jp * sr[:, None, None], r * sr[:, None]

    def total(J, idx, n):
        t = (J * r[..., None]).sum(1)
        return torch.zeros(n, t.shape[1], device=DEV, dtype=F64).index_add_(0, idx, t).reshape(-1)

    grad = torch.cat([total(je, c, len(s["extrinsics"])), total(ji, gi, len(s["intrinsics"])),
                      total(jp, pt, len(s["points"]))])
    return dict(je=je, ji=ji, jp=jp, grad=grad)


def _segments(v, tr, n):
    return torch.zeros((n,) + v.shape[1:], device=DEV, dtype=F64).index_add_(0, tr, v)


def _exact_tri_f32(case, seed):
    """N-view estimate (the smallest singular vector of the 3n x (4 + n)
    design, its n depths eliminated), then the Gauss-Newton steps."""
    P, _, tr, cam, xy = _track_scene(case, seed)
    P, xy, nt = P.float().double(), xy.float().double(), case["tracks"]
    Pc = P[cam]
    xt = torch.cat([xy, torch.ones_like(xy[:, :1])], 1)
    c2 = (xt * xt).sum(1)
    q = (xt[:, None, :] @ Pc)[:, 0]  # P^T x~: c h
    PtP = _segments(Pc.transpose(1, 2) @ Pc, tr, nt)
    qq = q[:, :, None] * q[:, None, :]
    lam = torch.zeros(nt, device=DEV, dtype=F64)
    eye = torch.eye(4, device=DEV, dtype=F64)
    A = PtP - _segments(qq / c2[:, None, None], tr, nt)
    Xh = torch.ones(nt, 4, 1, device=DEV, dtype=F64)
    for _ in range(3):
        # (P^T P - sum q q^T / c^2) X = lam (I + sum q q^T / (c^2 (c^2 - lam))) X,
        # the smallest lam by inverse iteration
        G = eye + _segments(qq / (c2 * (c2 - lam[tr]))[:, None, None], tr, nt)
        for _ in range(20):
            Xh = torch.linalg.solve(A, G @ Xh)
            Xh = Xh / Xh.norm(dim=1, keepdim=True)
        lam = ((Xh.transpose(1, 2) @ A @ Xh) / (Xh.transpose(1, 2) @ G @ Xh)).reshape(-1)
    Xh = Xh[..., 0]
    X = Xh[:, :3] / Xh[:, 3:]

    def project(X):
        h = (Pc[:, :, :3] @ X[tr][..., None])[..., 0] + Pc[:, :, 3]
        return h, h[:, :2] / h[:, 2:]

    live = torch.ones(nt, dtype=torch.bool, device=DEV)
    for _ in range(case["steps"]):
        h, u = project(X)
        res = u - xy
        J = (Pc[:, :2, :3] - u[..., None] * Pc[:, 2:, :3]) / h[:, 2][:, None, None]
        H = _segments(J.transpose(1, 2) @ J, tr, nt)
        gr = _segments((J * res[..., None]).sum(1), tr, nt)
        e0 = _segments((res * res).sum(1), tr, nt)
        Xn = X - torch.linalg.solve(H, gr)
        e1 = _segments(((project(Xn)[1] - xy) ** 2).sum(1), tr, nt)
        live = live & (e1 <= e0)
        X = torch.where(live[:, None], Xn, X)
    z = project(X)[0][:, 2]
    depth = torch.full((nt,), math.inf, device=DEV, dtype=F64).scatter_reduce_(0, tr, z, "amin")
    return dict(X=X, status=None, depth=depth)


def _exact_pack(case, seed):
    a = _pack_scene(case, seed)
    rec = a["reconstructed"].bool()
    nc = int(rec.sum())
    ext = torch.zeros(len(rec), 6, dtype=F64, device=DEV)
    ext[:nc] = torch.cat([_angle_axis(a["cameras"][:, :9].reshape(-1, 3, 3)), a["cameras"][:, 9:12]], 1)[rec]
    img = a["track_image"].long()
    keep = rec[img]
    at = a["feature_offsets"][img[keep]] + a["track_feature"].long()[keep]
    obs = torch.zeros(len(img), 2, dtype=F64, device=DEV)
    obs[:len(at)] = a["features"][at].double()
    return dict(extrinsics=ext, intrinsics=a["group_intrinsics"], points=a["points"], observations=obs,
                camera_constant=None, camera_index=None, intrinsic_index=None, point_index=None, camera_image=None,
                counts=None)


def _exact_acransac(case, seed):
    x, X, models = _resection(case, seed)
    n, s = case["points"], 6
    h = models.reshape(-1, 1, 3, 4) @ torch.cat([X, torch.ones_like(X[:, :1])], 1)[None, :, :, None]
    h = h[..., 0]
    e = torch.sort(((h[..., :2] / h[..., 2:] - x) ** 2).sum(-1), dim=1).values
    lg = np.concatenate([[0.0], np.log10(np.arange(1, n + 1, dtype=np.float64))])
    fact = np.cumsum(lg)
    k = np.arange(s + 1, n + 1)
    tab = (fact[n] - fact[k] - fact[n - k]).astype(np.float32).astype(np.float64) + \
        (fact[k] - fact[s] - fact[k - s]).astype(np.float32).astype(np.float64)
    kk = torch.from_numpy(k).to(DEV)
    v = math.log10(n - s) + (math.log10(math.pi) + torch.log10(e[:, s:] + 1.1754943508222875e-38)) * (kk - s) + \
        torch.from_numpy(tab).to(DEV)
    best = v.min(1)
    return dict(nfa=best.values, error_max=e.gather(1, kk[best.indices][:, None] - 1)[:, 0], inliers=None, order=None)

"""gbba_launch_count counts kernels that were launched: between solves of two and
of four LM iterations it grows by as many as a trace of the device shows (the
set-up, whose library sorts are counted by a fixed number, is the same in
both).  FP64 below and above 16,384 observations, mixed, shared groups."""
import pytest

pytestmark = pytest.mark.gpu


def kernels(handle, abi, sc, opts):
    import torch
    for _ in range(4):  # (a process's first trace may come back empty)
        hp = abi.HostProblem(sc)
        torch.cuda.synchronize()
        before = handle.lib.gbba_launch_count(handle.h)
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            s = handle.solve(hp, opts)
            torch.cuda.synchronize()
        traced = sum(1 for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA
                     and not e.name.lower().startswith(("memcpy", "memset")))
        if traced > 0:
            return s, handle.lib.gbba_launch_count(handle.h) - before, traced
    pytest.skip("the device gives no trace of its kernels")


@pytest.mark.parametrize("graphs", [0, 1])
@pytest.mark.parametrize("kind", ["fp64", "fp64 many", "mixed", "shared"])
def test_iterations_count_what_they_launch(kind, graphs, handle, abi, scenes):
    sc = scenes.medium_scene(num_cameras=12, num_points=4000 if kind == "fp64 many" else 600, mean_views=5, seed=961,
                             hold=(0, 1))
    if kind == "shared":
        sc["intrinsic_index"] = sc["intrinsic_index"] * 0
        sc["intrinsics"] = sc["intrinsics"][:1]
    assert (len(sc["observations"]) >= 16384) == (kind == "fp64 many")
    counts = []
    for n in (2, 4):
        opts = scenes.ba_options_for(sc, max_num_iterations=n, use_cuda_graphs=graphs, fp64_polish_iterations=0,
                                     function_tolerance=0.0, gradient_tolerance=0.0, parameter_tolerance=0.0,
                                     precision=abi.PRECISION_MIXED if kind == "mixed" else abi.PRECISION_FP64)
        handle.solve(abi.HostProblem(sc), opts)  # (allocations and attributes)
        s, counted, traced = kernels(handle, abi, sc, opts)
        assert s.num_iterations == n and s.num_successful_steps > 0
        counts.append((counted, traced))
    assert counts[1][0] - counts[0][0] == counts[1][1] - counts[0][1]

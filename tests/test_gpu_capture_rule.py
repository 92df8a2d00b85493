"""GPU: which calls replay a captured step. Launches of graphs are counted with the
profiler's trace of the CUDA runtime."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def graph_launches(call):
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    counts = {}
    for ev in p.events():
        counts[ev.name] = counts.get(ev.name, 0) + 1
    if not any(k.startswith(("cudaLaunchKernel", "cuLaunchKernel", "cudaGraphLaunch", "cuGraphLaunch")) for k in counts):
        pytest.skip("the profiler records no runtime calls here")
    return max(counts.get("cudaGraphLaunch", 0), counts.get("cuGraphLaunch", 0))


@pytest.mark.parametrize("steps", [31, 32, 100])
def test_a_long_call_is_captured_at_once_in_segments_or_not(nb, steps):
    """nbody_forward_checkpointed steps in segments of ceil(sqrt(steps)); they are one call."""
    pos, vel, mass = nb.generate(600, gen_type=1, seed=1)
    want = steps if steps >= 32 else 0
    torch.zeros(1, device="cuda")
    for call in ("step", "forward_checkpointed"):
        with nb.Engine() as e:
            e.set_particles(pos, vel, mass)
            assert graph_launches(lambda: getattr(e, call)(steps)) == want, call
            e.set_particles(pos, vel, mass)
            assert graph_launches(lambda: getattr(e, call)(steps)) == steps, call

"""The FP16 half-sweep takes two or four leaves per thread by the grid's size and by whether the call waits
for its work (host arrays): the same values to the bit, at the sizes on both sides of the limits and with
a last group that is not full."""
import numpy as np
import pytest

from hnanosolver_b200 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaves", [4399, 4400, 4401, 5999, 6001])
def test_host_call_equals_device_call(leaves):
    from hnanosolver_b200 import lib as hl

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    o = np.ascontiguousarray(synth.sort_leaves_nanovdb(synth._box_leaves(152))[:leaves])
    a, b, c = (hl.Grid(o, voxel_size=0.1) for _ in range(3))
    n = a.num_voxels
    gen = torch.Generator(device="cuda").manual_seed(4)
    vel = torch.randn((n, 3), device="cuda", generator=gen).bfloat16()
    desc = hl.MixedDesc(dt=0.05, omega=1.6, tolerance=1e-12, max_outer=2, inner_iterations=6, flags=0)
    out, persistent = torch.empty_like(vel), torch.empty_like(vel)
    c.set_option(hl.OPT_SPLIT_SOLVE, hl.SPLIT_PERSISTENT)  # four leaves per thread at every size
    torch.cuda.synchronize()
    a.step_mixed(vel, out, [], [], desc)
    c.step_mixed(vel, persistent, [], [], desc)
    host = vel.float().cpu().numpy()
    b.step_mixed_host(host, [], desc)
    a.synchronize(), c.synchronize()
    assert torch.isfinite(out.float()).all() and torch.equal(out, persistent)
    assert torch.equal(out.float().cpu(), torch.from_numpy(host))
    for g in (a, b, c):
        g.close()

"""HNS_OPT_WAIT_POLLS on the solve held in shared memory: the poll limit is the option's value (a poll
is a load from L2, at least 200 cycles of at most 2 GHz, so 2^16 of them take 6 ms or more; at the first
poll the solve gives up within microseconds), however large the value, and the context recovers."""
import pytest

from hnanosolver_b200 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("polls,least_ms", [(0, 0.0), (1 << 16, 6.0), (0x7FFFFFFF, 100.0)])
def test_gives_up_after_that_many_polls(polls, least_ms):
    from hnanosolver_b200 import lib as hl

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    grid = hl.Grid(synth.spheres_topology(96, 3, 8.0, 20.0, seed=12), voxel_size=0.1)
    stream = torch.cuda.Stream()
    grid.set_stream(stream.cuda_stream)
    div = torch.randn(grid.num_voxels, device="cuda")
    p, q = torch.zeros_like(div), torch.zeros_like(div)
    torch.cuda.synchronize()
    grid.rbgs(div, q, 8, 1.5, hl.SOLVE_ZERO_INIT)
    grid.device_status()
    grid.set_option(hl.OPT_WAIT_POLLS, polls)
    a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    a.record(stream)
    grid.rbgs(div, p, 8, 1.5, hl.SOLVE_ZERO_INIT)
    b.record(stream)
    assert hl.lib.hns_device_status(grid.handle) == 8  # HNS_ERR_TIMEOUT
    assert a.elapsed_time(b) >= least_ms
    grid.set_option(hl.OPT_WAIT_POLLS, -1)
    grid.rbgs(div, p, 8, 1.5, hl.SOLVE_ZERO_INIT)
    grid.device_status()
    assert torch.equal(p, q)
    grid.close()

"""A call that a CUDA error ended does not make the next one fail: the runtime keeps the last error until
it is read, and the launches of a later call must not read an earlier call's."""
import pytest

from hnanosolver_b200 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_next_call_after_a_refused_one():
    """A call that waits (info) on a stream that its caller is capturing is refused by CUDA."""
    from cuda.bindings import runtime as rt

    from hnanosolver_b200 import lib as hl

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    grid = hl.Grid(synth.spheres_topology(64, 2, 8.0, 16.0, seed=3), voxel_size=0.1)
    vel = torch.randn((grid.num_voxels, 3), device="cuda")
    div, want = torch.empty(grid.num_voxels, device="cuda"), torch.empty(grid.num_voxels, device="cuda")
    torch.cuda.synchronize()
    grid.project(vel.clone(), 8, 1.5, info=True)  # makes the scratch
    grid.divergence(vel, want)
    grid.synchronize()
    err, stream = rt.cudaStreamCreateWithFlags(rt.cudaStreamNonBlocking)
    assert int(err) == 0
    grid.set_stream(int(stream))
    assert int(rt.cudaStreamBeginCapture(stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeRelaxed)[0]) == 0
    with pytest.raises(hl.HnsError):
        grid.project(vel, 8, 1.5, info=True)
    rt.cudaStreamEndCapture(stream)  # invalidated: no graph
    grid.divergence(vel, div)
    grid.synchronize()
    assert torch.equal(div, want)
    grid.set_stream(0)
    grid.close()
    assert int(rt.cudaStreamDestroy(stream)[0]) == 0

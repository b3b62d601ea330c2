"""The library's own graphs (a checked FP32 solve's loop, a multigrid refinement's spare iterations) are
captured on the context's own stream, not on the caller's: a context that works on the default stream has
them too, and a caller's blocking stream does not refuse other threads' work on the default stream while
a graph is made."""
import ctypes
import threading

import pytest

from hnanosolver_b200 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

LEGACY_STREAM = 1  # cudaStreamLegacy


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda", 0)


def _solver(dev, stream):
    from hnanosolver_b200 import lib as hl

    grid = hl.Grid(synth.spheres_topology(96, 3, 8.0, 20.0, seed=12), voxel_size=0.1)
    grid.set_option(hl.OPT_SPLIT_SOLVE, hl.SPLIT_PER_COLOUR)
    if stream:
        grid.set_stream(stream)
    gen = torch.Generator(device=dev).manual_seed(5)
    vel = torch.randn((grid.num_voxels, 3), device=dev, generator=gen)
    out = torch.empty_like(vel)

    def step(every):
        grid.step_plain(vel, out, [], [], hl.StepDesc(dt=0.1, max_iterations=120, omega=1.7, tolerance=1e-9,
                                                      check_every=every, flags=0))
        grid.synchronize()
        return out.clone()

    torch.cuda.synchronize()
    return grid, step


def test_loop_on_the_default_stream(dev):
    own, legacy = _solver(dev, None), _solver(dev, LEGACY_STREAM)
    counts = []
    for grid, step in (own, legacy):
        step(10)
        grid.profile_read()
        got = step(10)
        counts.append(grid.profile_read().kernel_launches)
        assert torch.isfinite(got).all()
    assert counts[0] == counts[1] < 60  # not the 240 half-sweeps of launches
    assert torch.equal(own[1](10), legacy[1](10))
    own[0].close(), legacy[0].close()


def test_other_threads_keep_the_default_stream(dev):
    stream = ctypes.c_void_p()
    assert int(torch.cuda.cudart().cudaStreamCreate(ctypes.addressof(stream))) == 0  # a blocking stream
    grid, step = _solver(dev, stream.value)
    ref_grid, ref = _solver(dev, None)
    stop, errors, done = threading.Event(), [], []

    def other():
        x = torch.zeros(1024, device=dev)
        while not stop.is_set():
            try:
                x.add_(1.0)
                done.append(1)
            except Exception as e:  # noqa: BLE001
                errors.append(e)
                return

    t = threading.Thread(target=other)
    t.start()
    try:
        got = [step(every) for every in range(4, 40, 2)]  # a graph each
    finally:
        stop.set()
        t.join()
    assert done and not errors
    for every, g in zip(range(4, 40, 2), got):
        assert torch.equal(g, ref(every))
    torch.cuda.synchronize()
    grid.close(), ref_grid.close()
    assert int(torch.cuda.cudart().cudaStreamDestroy(stream.value)) == 0

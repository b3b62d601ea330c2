"""A checked FP32 solve, whose iterations after the first check run as a device-side loop: it stops at
the first check within the tolerance, or at the cap, with the values of that many iterations without
checks, to the bit. Intervals that divide the cap and that do not, one check, several, none passing."""
import pytest

from hnanosolver_b200 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda", 0)


@pytest.mark.parametrize("split", ["AUTO", "PER_COLOUR"])
@pytest.mark.parametrize("cap,every,tolerance", [(60, 10, 0.5), (60, 10, 0.05), (200, 6, 0.01), (50, 20, 1e-9), (10, 10, 1e-9),
                                                 (24, 10, 1e-9), (8, 20, 1e-9)])
def test_stops_with_the_values_of_as_many_iterations(dev, cap, every, tolerance, split):
    from hnanosolver_b200 import lib as hl

    o = synth.spheres_topology(96, 3, 8.0, 20.0, seed=12)
    grid = hl.Grid(o, voxel_size=0.1)
    grid.set_option(hl.OPT_SPLIT_SOLVE, getattr(hl, "SPLIT_" + split))
    g = torch.Generator(device=dev).manual_seed(5)
    vel = torch.randn((grid.num_voxels, 3), device=dev, generator=g)

    def step(iterations, tol, check):
        out = torch.empty_like(vel)
        torch.cuda.synchronize()
        desc = hl.StepDesc(dt=0.1, max_iterations=iterations, omega=1.7, tolerance=tol, check_every=check, flags=0)
        try:
            ran = grid.step_plain(vel, out, [], [], desc, info=True).iterations
        except hl.HnsError as e:
            assert e.status == 6 and tol == 1e-9  # not converged at the cap
            ran = iterations
        grid.synchronize()
        return out, ran

    for _ in range(2):  # the second call runs the graph that the first made
        got, ran = step(cap, tolerance, every)
        assert 0 < ran <= cap and (ran < cap or tolerance < 1e-6)
        want, _ = step(ran, 0.0, 0)
        assert torch.equal(got, want)

"""The graph of a checked FP32 solve's loop serves every tolerance and iteration cap, and a program that
solves with another factor omega each time makes no graph per solve. Seen in the count of launches, in
which those captured into a new graph are included; the values are those of unchecked iterations."""
import pytest

from hnanosolver_b200 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_graphs_are_made_once():
    from hnanosolver_b200 import lib as hl

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    grid = hl.Grid(synth.spheres_topology(96, 3, 8.0, 20.0, seed=12), voxel_size=0.1)
    grid.set_option(hl.OPT_SPLIT_SOLVE, hl.SPLIT_PER_COLOUR)
    gen = torch.Generator(device="cuda").manual_seed(5)
    vel = torch.randn((grid.num_voxels, 3), device="cuda", generator=gen)
    every = 10

    def solve(omega, tolerance, cap):
        """Launches of a step's solve, whose result must be that of as many iterations without checks."""
        out, want = torch.empty_like(vel), torch.empty_like(vel)
        torch.cuda.synchronize()
        grid.profile_read()
        grid.step_plain(vel, out, [], [], hl.StepDesc(dt=0.1, max_iterations=cap, omega=omega, tolerance=tolerance,
                                                      check_every=every, flags=0))
        count = grid.profile_read().kernel_launches
        ran = grid.last_solve().iterations
        grid.step_plain(vel, want, [], [], hl.StepDesc(dt=0.1, max_iterations=ran, omega=omega, tolerance=0.0,
                                                       check_every=0, flags=0))
        grid.synchronize()
        assert torch.equal(out, want)
        return count

    first = solve(1.7, 1e-2, 100)
    repeated = solve(1.7, 1e-2, 100)
    assert first > repeated  # the tables, and the loop's body captured
    # Check 0's launches and the loop's own, whatever the tolerance and the cap.
    assert repeated < 3 * every + 20
    for tolerance, cap in ((1e-3, 100), (1e-1, 100), (1e-9, 200), (1e-9, 60)):
        assert solve(1.7, tolerance, cap) == repeated
    # Other factors, each once: launches for every iteration, nothing captured.
    plain = [solve(1.3 + 0.01 * k, 1e-9, 100) for k in range(4)]
    assert len(set(plain)) == 1 and plain[0] >= 200
    # One that comes again gets its graph, and then keeps it.
    assert solve(1.3, 1e-9, 100) > repeated
    assert solve(1.3, 1e-9, 100) == repeated == solve(1.7, 1e-9, 100)
    grid.close()

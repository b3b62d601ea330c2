"""Refined solves of velocities so small that a residual's scale leaves FP32's normal numbers: the results
are finite and no larger than the input (a projection does not enlarge the velocity's norm; here by less
than a tenth), in every form of the inner solve."""
import pytest

from hnanosolver_b200 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [1e-30, 1e-33, 1e-35, 1e-37, 1e-38])
@pytest.mark.parametrize("form", ["rows", "packed", "split", "multigrid", "fp32", "fp32_multigrid"])
def test_finite(form, size):
    from hnanosolver_b200 import lib as hl

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    grid = hl.Grid(synth.spheres_topology(64, 3, 6.0, 14.0, seed=9), voxel_size=0.1)
    gen = torch.Generator(device="cuda").manual_seed(2)
    vel = torch.randn((grid.num_voxels, 3), device="cuda", generator=gen).clamp(-3.0, 3.0) * size
    vel[::7] = 0.0
    if form.startswith("fp32"):
        out = torch.empty_like(vel)
        flags = hl.SOLVE_REFINE | (hl.SOLVE_MULTIGRID if form.endswith("multigrid") else 0)
        torch.cuda.synchronize()
        grid.step_plain(vel, out, [], [], hl.StepDesc(dt=0.0, max_iterations=0, omega=1.6, tolerance=1e-6, check_every=0,
                                                      flags=flags, max_outer=8, inner_iterations=20))
    else:
        layouts = {"rows": hl.INNER_ROWS, "packed": hl.INNER_PACKED}
        grid.set_option(hl.OPT_INNER_LAYOUT, layouts.get(form, hl.INNER_SPLIT))
        vel = vel.bfloat16()
        out = torch.empty_like(vel)
        multigrid = form == "multigrid"
        torch.cuda.synchronize()
        grid.step_mixed(vel, out, [], [], hl.MixedDesc(dt=0.0, omega=1.6, tolerance=1e-6, max_outer=8,
                                                       inner_iterations=2 if multigrid else 20,
                                                       flags=hl.SOLVE_MULTIGRID if multigrid else 0))
    grid.synchronize()
    assert torch.isfinite(out).all()
    scale = 1.0 / size
    assert (out.double() * scale).norm() <= 1.1 * (vel.double() * scale).norm()
    grid.close()

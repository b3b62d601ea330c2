"""The shared-memory tiles of the multi-field advection and the row kernels, at the sizes, field counts,
trace lengths and alignments where their paths part.

  * FP32 fields against the FP32 oracle, 1 to 7 fields (one pass takes five), traces inside the
    tile, across it, and out of the domain. The sums of a tap differ from the oracle's by rounding,
    at most 8 2^-24 of the largest velocity; on a trace of 40 voxels that moves the forward tap by
    2e-5 voxels, or 4e-5 of the field's maximum at its steepest: bound 1e-4.
  * FP16 fields along a BF16 velocity (the last pass of hns_advance_mixed): the FP32 operations on
    widened values and one rounding, so exactly the FP32 entry's result rounded to FP16.
  * Arrays that vector loads cannot take give the values of aligned ones to the bit."""
import numpy as np
import pytest

from conftest import rel_err
from hnanosolver_b200 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

NAMES = ("temperature", "density", "fuel", "waste", "flame")


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda", 0)


def _origins(name):
    if name == "one":
        return np.array([[-8, 0, 16]], np.int32)
    o = synth.spheres_topology(64, 3, 6.0, 14.0, seed=9)
    return np.ascontiguousarray(np.random.default_rng(1).permutation(o))


def _fields(n, dev, count, speed, seed=3):
    g = torch.Generator(device=dev).manual_seed(seed)
    vel = speed * torch.randn((n, 3), device=dev, generator=g)
    return vel, [torch.randn(n, device=dev, generator=g) for _ in range(count)]


@pytest.mark.parametrize("speed", [0.5, 5.0, 20.0])
@pytest.mark.parametrize("count", [1, 2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("name", ["one", "spheres"])
def test_fp32_fields_against_the_oracle(dev, oracle, name, count, speed):
    from hnanosolver_b200 import lib as hl

    o = _origins(name)
    grid, t = hl.Grid(o, voxel_size=0.1), oracle.topo(o)
    vel, fields = _fields(grid.num_voxels, dev, count, speed)
    outs = [torch.empty_like(f) for f in fields]
    torch.cuda.synchronize()
    dt = 1.0 / 24.0
    grid.advect_scalars(vel, fields, outs, dt)
    grid.synchronize()
    want = t.advect_scalars(vel.cpu().numpy(), [f.cpu().numpy() for f in fields], dt, 10.0)
    for a, b in zip(outs, want):
        assert rel_err(a.cpu().numpy(), b) <= 1e-4


def _params(hl, **kw):
    from oracle.binding import CombustionParams as OP

    p = OP.houdini_defaults()
    p.vorticityScale, p.factorScale, p.disturbanceEnable, p.gravity, p.substeps = 0.3, 1.0, 0.0, 0.0, 1
    for k, v in kw.items():
        setattr(p, k, v)
    return hl.CombustionParams.from_buffer_copy(bytes(p))


def _mixed(hl, grid, fin, fout, combustion=2, factor=1.0):
    model = hl.ForceModel(combustion=combustion, burn_rate=0.5, heat_release=1.0, ignition_temp=0.0, density_buoyancy=0.0)
    desc = hl.MixedDesc(dt=0.0, omega=1.9, tolerance=1e-3, max_outer=2, inner_iterations=10, flags=0)
    torch.cuda.synchronize()
    grid.advance_mixed(fin, fout, None, 1.0 / 24.0, _params(hl, factorScale=factor), model, desc)
    grid.synchronize()


def _half_state(n, dev, count, speed):
    vel, fields = _fields(n, dev, count, speed)
    return {"velocity": vel.bfloat16(), **{k: f.half() for k, f in zip(NAMES, fields)}}


@pytest.mark.parametrize("speed", [0.5, 5.0, 20.0])
@pytest.mark.parametrize("count", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("name", ["one", "spheres"])
def test_fp16_fields_are_the_fp32_ones_rounded(dev, name, count, speed):
    from hnanosolver_b200 import lib as hl

    grid = hl.Grid(_origins(name), voxel_size=0.1)
    fin = _half_state(grid.num_voxels, dev, count, speed)
    fout = {k: torch.empty_like(v) for k, v in fin.items()}
    _mixed(hl, grid, fin, fout)
    f32 = [fin[k].float() for k in NAMES[:count]]
    outs = [torch.empty_like(f) for f in f32]
    vel = fout["velocity"].float()
    torch.cuda.synchronize()
    grid.advect_scalars(vel, f32, outs, 1.0 / 24.0)
    grid.synchronize()
    for k, want in zip(NAMES, outs):
        assert torch.equal(fout[k], want.half()), k


def test_outputs_that_are_other_fields_inputs(dev):
    from hnanosolver_b200 import lib as hl

    grid = hl.Grid(_origins("spheres"), voxel_size=0.1)
    fin = _half_state(grid.num_voxels, dev, 5, 2.0)
    want = {k: torch.empty_like(v) for k, v in fin.items()}
    _mixed(hl, grid, fin, want)
    swapped = dict(want, velocity=torch.empty_like(fin["velocity"]), temperature=torch.empty_like(fin["temperature"]),
                   density=fin["fuel"], fuel=fin["waste"], waste=fin["density"], flame=torch.empty_like(fin["flame"]))
    _mixed(hl, grid, fin, swapped)
    for k in fin:
        assert torch.equal(swapped[k], want[k]), k


def _shifted(t):
    """The values of t one element past an aligned address."""
    s = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].view(t.shape)
    return s.copy_(t)


@pytest.mark.parametrize("factor", [-1.0, 0.0, 1.0])
@pytest.mark.parametrize("combustion", [0, 1, 2])
def test_unaligned_fire_arrays(dev, combustion, factor):
    from hnanosolver_b200 import lib as hl

    grid = hl.Grid(_origins("spheres"), voxel_size=0.1)
    fin = _half_state(grid.num_voxels, dev, 5, 2.0)
    a = {k: torch.empty_like(v) for k, v in fin.items()}
    b = {k: _shifted(v) for k, v in fin.items()}
    _mixed(hl, grid, fin, a, combustion, factor)
    _mixed(hl, grid, {k: _shifted(v) for k, v in fin.items()}, b, combustion, factor)
    for k in a:
        assert torch.equal(a[k], b[k]), k


@pytest.mark.parametrize("walls", [False, True])
@pytest.mark.parametrize("name", ["one", "spheres"])
def test_unaligned_fp32_arrays(dev, name, walls):
    from hnanosolver_b200 import lib as hl

    grid = hl.Grid(_origins(name), voxel_size=0.1)
    vel, (p, dens) = _fields(grid.num_voxels, dev, 2, 2.0)
    desc = hl.StepDesc(dt=1.0 / 24.0, max_iterations=6, omega=1.7, tolerance=0.0, check_every=0, flags=hl.SOLVE_NEUMANN if walls else 0)
    got = []
    for move in (torch.clone, _shifted):
        v, q, d = move(vel), move(p), move(dens)
        div, out, sv, sd = move(p), move(vel), move(vel), move(p)
        torch.cuda.synchronize()
        grid.divergence(v, div)
        grid.subtract_gradient(v, q, out)
        grid.step_plain(v, sv, [d], [sd], desc)
        grid.synchronize()
        got.append((div, out, sv, sd))
    for x, y in zip(*got):
        assert torch.equal(x, y)


@pytest.mark.parametrize("name", ["one", "corner", "spheres"])
def test_multigrid_on_small_and_shuffled_grids(dev, name):
    """The level transfers where every side of a leaf is missing, where two leaves touch at a corner only,
    and where neighbours lie anywhere in the order: a transfer that reads a wrong cell does not
    converge in the cycles that the sorted grids need (at most 12 refinements of two)."""
    from hnanosolver_b200 import lib as hl

    o = np.array([[0, 0, 0], [8, 8, 8]], np.int32) if name == "corner" else _origins(name)
    grid = hl.Grid(o, voxel_size=0.1)
    vel, (d,) = _fields(grid.num_voxels, dev, 1, 2.0)
    v, d = vel.bfloat16(), d.half()
    vo, do = torch.empty_like(v), torch.empty_like(d)
    torch.cuda.synchronize()
    info = grid.step_mixed(v, vo, [d], [do], hl.MixedDesc(dt=0.1, omega=1.9, tolerance=1e-5, max_outer=12, inner_iterations=2,
                                                          flags=hl.SOLVE_MULTIGRID), info=True)
    assert info.residual <= 1e-5

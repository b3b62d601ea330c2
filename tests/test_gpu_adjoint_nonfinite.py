"""Infinities and NaN that no adjoint reaches. Where the adjoint of an output is 0, the values that
output was computed from do not enter the gradient, finite or not (a loss over part of a domain whose
rest has blown up): the gradient is that of the same fields with the non-finite values replaced by 0."""
import numpy as np
import pytest

from hnanosolver_b200 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda", 0)


BAD = [float("nan"), float("inf"), -float("inf")]


def _grid(dev):
    """A grid, the slots of a few of its voxels and the mask of the voxels within 4 of one."""
    from hnanosolver_b200 import lib as hl

    o = synth.spheres_topology(64, 3, 6.0, 14.0, seed=9)
    ijk = torch.from_numpy(synth.leaf_dense_coords(o)).to(dev)
    slots = torch.from_numpy(np.random.default_rng(2).choice(len(ijk), 6, replace=False)).to(dev)
    near = torch.zeros(len(ijk), dtype=torch.bool, device=dev)
    for s in slots:
        near |= (ijk - ijk[s]).abs().amax(dim=1) <= 4
    return hl.Grid(o, voxel_size=0.1), slots, near


@pytest.mark.parametrize("factor", [1.0, -1.0])
@pytest.mark.parametrize("bad", BAD)
def test_confinement(dev, bad, factor):
    grid, slots, near = _grid(dev)
    gen = torch.Generator(device=dev).manual_seed(4)
    vel = torch.randn((grid.num_voxels, 3), device=dev, generator=gen)
    out_bar = torch.randn(vel.shape, device=dev, generator=gen)
    out_bar[near] = 0.0
    got = []
    for value in (bad, 0.0):
        vel[slots, 1] = value
        bar = torch.zeros_like(vel)
        torch.cuda.synchronize()
        grid.adjoint_vorticity_confinement(vel, out_bar, bar, 0.1, 0.4, factor)
        grid.synchronize()
        got.append(bar)
    assert torch.isfinite(got[0]).all() and torch.equal(got[0], got[1])
    grid.close()


@pytest.mark.parametrize("bad", BAD)
def test_scalar_beside_a_velocity_with_adjoints(dev, bad):
    """The scalar's gradient of a step whose velocity has adjoints everywhere, its own being 0 near the
    bad voxels. A trace from a NaN starts in the cell at the origin, which the box holds. Sums by atomics
    in any order: of fewer than 200 terms (the voxels whose traces reach one), each at most 5, so within
    200^2 2^-24 5 = 0.012; a missing or an extra term is of the order of 1."""
    from hnanosolver_b200 import lib as hl

    o = synth.sort_leaves_nanovdb(synth._box_leaves(32))
    grid = hl.Grid(o, voxel_size=0.1)
    ijk = torch.from_numpy(synth.leaf_dense_coords(o)).to(dev)
    slots = torch.from_numpy(np.random.default_rng(2).choice(len(ijk), 6, replace=False)).to(dev)
    gen = torch.Generator(device=dev).manual_seed(4)
    n = grid.num_voxels
    vel = torch.rand((n, 3), device=dev, generator=gen) - 0.5
    dens = torch.randn(n, device=dev, generator=gen)
    vel_out_bar = torch.randn((n, 3), device=dev, generator=gen)
    dens_out_bar = torch.randn(n, device=dev, generator=gen).clamp(-5.0, 5.0)
    for s in slots:
        dens_out_bar[(ijk - ijk[s]).abs().amax(dim=1) <= 4] = 0.0
    got = []
    for value in (bad, 0.0):
        vel[slots, 1] = value
        vel_bar, dens_bar = torch.zeros_like(vel), torch.zeros_like(dens)
        torch.cuda.synchronize()
        grid.adjoint_step_plain(vel, [dens], vel_out_bar, [dens_out_bar], vel_bar, [dens_bar], 0.1, 4, 1.0)
        grid.synchronize()
        got.append(dens_bar)
    assert torch.isfinite(got[0]).all()
    assert (got[0] - got[1]).abs().max() <= 0.012
    grid.close()


@pytest.mark.parametrize("bad", BAD[:1])
def test_velocity_beside_a_scalar_with_adjoints(dev, bad):
    """A scalar's adjoint next to a bad velocity: its forward trace ends at NaN, in the cell at the origin,
    where the velocity's own adjoint is 0 and stays so (bit for bit: nothing else reaches that corner)."""
    from hnanosolver_b200 import lib as hl

    o = synth.sort_leaves_nanovdb(synth._box_leaves(32))
    grid = hl.Grid(o, voxel_size=0.1)
    ijk = torch.from_numpy(synth.leaf_dense_coords(o)).to(dev)
    at = (ijk == torch.tensor([21, 13, 18], device=dev, dtype=ijk.dtype)).all(dim=1)
    vel = torch.full((grid.num_voxels, 3), 0.3, device=dev)
    vel[at] = bad
    dens = torch.rand(grid.num_voxels, device=dev, generator=torch.Generator(device=dev).manual_seed(4))
    out_bar = (((ijk - ijk[at]).abs().amax(dim=1) <= 2) & ~at).float()
    dens_bar, vel_bar = torch.zeros_like(dens), torch.zeros_like(vel)
    torch.cuda.synchronize()
    grid.adjoint_advect_scalar(vel, dens, out_bar, dens_bar, vel_bar, 0.1)
    grid.synchronize()
    corner = (ijk <= 8).all(dim=1)
    assert (vel_bar[corner] == 0.0).all()
    grid.close()


def test_fire_fields_after_a_bad_velocity_source(dev):
    """The fire step's scalars are advected back together. A velocity source with a NaN in it makes the
    projected velocity NaN around it, which spoils the gradients of the fields that have adjoints, not those
    of fields whose adjoints are 0, one in each place of the records."""
    from hnanosolver_b200 import lib as hl

    o = synth.sort_leaves_nanovdb(synth._box_leaves(32))
    grid = hl.Grid(o, voxel_size=0.1)
    n = grid.num_voxels
    gen = torch.Generator(device=dev).manual_seed(4)
    names = ("density", "temperature", "fuel", "waste", "flame")
    fields = {k: torch.rand(n, device=dev, generator=gen) for k in names}
    fields["velocity"] = torch.rand((n, 3), device=dev, generator=gen)
    source = torch.zeros((n, 3), device=dev)
    source[n // 2] = float("nan")
    p = hl.CombustionParams()
    p.vorticityScale, p.factorScale, p.substeps = 0.3, 1.0, 1
    model = hl.ForceModel(combustion=2, burn_rate=0.0, heat_release=0.0, ignition_temp=0.0, density_buoyancy=0.0)
    for live in ("density", "flame"):
        out_bar = {k: torch.zeros(n, device=dev) for k in names}
        out_bar["velocity"] = torch.zeros((n, 3), device=dev)
        out_bar[live] = torch.randn(n, device=dev, generator=gen)
        in_bar = {k: torch.zeros_like(v) for k, v in fields.items()}
        torch.cuda.synchronize()
        grid.adjoint_advance(fields, {"velocity": source}, out_bar, in_bar, 0.1, 4, p, model)
        grid.synchronize()
        assert not torch.isfinite(in_bar[live]).all()
        for k in ("fuel", "waste", "flame"):  # the buoyancy gives the others the velocity's adjoint
            assert k == live or (in_bar[k] == 0.0).all(), (live, k)
    grid.close()

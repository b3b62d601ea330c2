"""The solve held in the SMs' shared memory (HNS_SPLIT_AUTO, the default where the grid fits) against
one launch per half-sweep (HNS_SPLIT_PER_COLOUR) and, for zero-gradient walls, the staged kernel:
the same arithmetic in the same order, so the same values to the bit. Grids: one leaf, fewer leaves
than SMs, a leaf more than a multiple of the SM count, several leaves per SM, sizes at which the
right-hand side no longer fits beside the values, and leaves in random order (every neighbour in
another CTA)."""
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


def _origins(name):
    if name == "one":
        return np.array([[-8, 0, 16]], np.int32)
    if name == "sms+1":  # 149 leaves of a slab
        return np.ascontiguousarray(synth._box_leaves(128)[:149])
    if name == "box160":  # 8,000 leaves: 55 per SM, the FP32 right-hand side streams
        return synth.sort_leaves_nanovdb(synth._box_leaves(160))
    o = synth.spheres_topology(96, 3, 8.0, 20.0, seed=12)
    return np.ascontiguousarray(np.random.default_rng(0).permutation(o)) if name == "shuffled" else o


GRIDS = ["one", "sms+1", "spheres", "shuffled", "box160"]


def _pair(hl, name, per_colour=None):
    a, b = (hl.Grid(_origins(name), voxel_size=0.1) for _ in range(2))
    a.set_option(hl.OPT_SPLIT_SOLVE, hl.SPLIT_AUTO)
    b.set_option(*(per_colour or (hl.OPT_SPLIT_SOLVE, hl.SPLIT_PER_COLOUR)))
    return a, b


def _field(n, dev, seed, comps=1):
    g = torch.Generator(device=dev).manual_seed(seed)
    return torch.randn((n, comps) if comps > 1 else n, device=dev, generator=g)


@pytest.mark.parametrize("walls", [False, True])
@pytest.mark.parametrize("iterations,zero", [(4, True), (17, True), (12, False)])
@pytest.mark.parametrize("name", GRIDS)
def test_rbgs_bit_exact(dev, name, iterations, zero, walls):
    from hnanosolver_b200 import lib as hl

    a, b = _pair(hl, name, (hl.OPT_RBGS_KERNEL, hl.RBGS_PLAIN) if walls else None)
    div, p0 = _field(a.num_voxels, dev, 1), _field(a.num_voxels, dev, 2)
    pa, pb = p0.clone(), p0.clone()
    torch.cuda.synchronize()
    flags = (hl.SOLVE_ZERO_INIT if zero else 0) | (hl.SOLVE_NEUMANN if walls else 0)
    for g, p in ((a, pa), (b, pb)):
        g.rbgs(div, p, iterations, 1.6, flags)
        g.device_status()
    assert torch.isfinite(pa).all() and torch.equal(pa, pb)
    a.close(), b.close()


@pytest.mark.parametrize("name", GRIDS)
def test_checked_and_mixed_solves_bit_exact(dev, name):
    from hnanosolver_b200 import lib as hl

    a, b = _pair(hl, name)
    n = a.num_voxels
    vel, dens = _field(n, dev, 3, 3), _field(n, dev, 4)
    step = hl.StepDesc(dt=0.05, max_iterations=120, omega=1.7, tolerance=1e-3, check_every=10, flags=0)
    mixed = hl.MixedDesc(dt=0.05, omega=1.7, tolerance=1e-5, max_outer=6, inner_iterations=20, flags=0)
    got = []
    for g in (a, b):
        vo, do = torch.empty_like(vel), torch.empty_like(dens)
        hv, hd = vel.bfloat16(), dens.half()
        ho, hs = torch.empty_like(hv), torch.empty_like(hd)
        torch.cuda.synchronize()
        g.step_plain(vel, vo, [dens], [do], step)
        solve = g.last_solve()
        g.step_mixed(hv, ho, [hd], [hs], mixed)
        p = torch.empty(n, dtype=torch.float64, device=dev)
        g.refine_pressure(p)
        g.device_status()
        got.append((vo, do, ho, hs, p, solve.iterations))
    for x, y in zip(*got):
        assert x == y if isinstance(x, int) else torch.equal(x, y)
    a.close(), b.close()


@pytest.mark.parametrize("name", ["one", "sms+1", "shuffled"])
def test_adjoint_rbgs_bit_exact(dev, name):
    from hnanosolver_b200 import lib as hl

    a, b = _pair(hl, name)
    p_bar, d0 = _field(a.num_voxels, dev, 5), _field(a.num_voxels, dev, 6)
    da, db = d0.clone(), d0.clone()
    torch.cuda.synchronize()
    for g, d in ((a, da), (b, db)):
        g.adjoint_rbgs(p_bar, d, 9, 1.4)
        g.device_status()
    assert torch.isfinite(da).all() and torch.equal(da, db)
    a.close(), b.close()


def test_wait_gives_up_then_recovers(dev):
    """The bounded wait for the other CTAs' faces, made to run out (HNS_OPT_WAIT_POLLS): the error
    flag is raised once, every CTA returns, and the next solve is clean."""
    from hnanosolver_b200 import lib as hl

    a, b = _pair(hl, "spheres")
    div = _field(a.num_voxels, dev, 7)
    pa, pb = torch.zeros_like(div), torch.zeros_like(div)
    torch.cuda.synchronize()
    a.set_option(hl.OPT_WAIT_POLLS, 0)
    a.rbgs(div, pa, 8, 1.5, hl.SOLVE_ZERO_INIT)
    assert hl.lib.hns_device_status(a.handle) == 8  # HNS_ERR_TIMEOUT
    a.device_status()
    a.set_option(hl.OPT_WAIT_POLLS, -1)
    for g, p in ((a, pa), (b, pb)):
        g.rbgs(div, p, 8, 1.5, hl.SOLVE_ZERO_INIT)
        g.device_status()
    assert torch.equal(pa, pb)
    a.close(), b.close()


@pytest.mark.parametrize("name", GRIDS)
def test_walls_per_colour_bit_exact(dev, name):
    """Zero-gradient walls, one launch per half-sweep on colour-split leaves against the staged
    kernel: fixed iterations from zero and from given values, and a checked solve's iterates."""
    from hnanosolver_b200 import lib as hl

    a, b = (hl.Grid(_origins(name), voxel_size=0.1) for _ in range(2))
    a.set_option(hl.OPT_SPLIT_SOLVE, hl.SPLIT_PER_COLOUR)
    b.set_option(hl.OPT_RBGS_KERNEL, hl.RBGS_PLAIN)
    n = a.num_voxels
    div, p0, vel = _field(n, dev, 8), _field(n, dev, 9), _field(n, dev, 10, 3)
    step = hl.StepDesc(dt=0.05, max_iterations=60, omega=1.5, tolerance=1e-2, check_every=10, flags=hl.SOLVE_NEUMANN)
    got = []
    for g in (a, b):
        p, q, vo = p0.clone(), torch.empty_like(p0), torch.empty_like(vel)
        torch.cuda.synchronize()
        g.rbgs(div, p, 5, 1.6, hl.SOLVE_NEUMANN)
        g.rbgs(div, q, 5, 1.6, hl.SOLVE_NEUMANN | hl.SOLVE_ZERO_INIT)
        g.step_plain(vel, vo, [], [], step)
        got.append((p, q, vo, g.last_solve().iterations))
    for x, y in zip(*got):
        assert x == y if isinstance(x, int) else torch.equal(x, y)
    a.close(), b.close()

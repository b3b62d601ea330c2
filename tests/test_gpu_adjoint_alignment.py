"""The transposed red-black sweeps on arrays that are only 4-byte aligned (views into a program's
larger buffer), by both launch forms: the values of aligned arrays, to the bit."""
import pytest

from hnanosolver_b200 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda", 0)


@pytest.mark.parametrize("form", ["AUTO", "PER_COLOUR"])
@pytest.mark.parametrize("shift", [(0, 1), (1, 0), (2, 3)])
def test_adjoint_rbgs_of_unaligned_arrays(dev, shift, form):
    from hnanosolver_b200 import lib as hl

    grid = hl.Grid(synth.spheres_topology(64, 3, 6.0, 14.0, seed=9), voxel_size=0.1)
    grid.set_option(hl.OPT_SPLIT_SOLVE, getattr(hl, "SPLIT_" + form))
    n = grid.num_voxels
    gen = torch.Generator(device=dev).manual_seed(5)
    p_bar, d0 = (torch.randn(n, device=dev, generator=gen) for _ in range(2))
    got = []
    for s in ((0, 0), shift):
        store = [torch.full((n + 8,), 7.0, device=dev) for _ in range(2)]
        p, d = (x[k:k + n] for x, k in zip(store, s))
        p.copy_(p_bar), d.copy_(d0)
        torch.cuda.synchronize()
        grid.adjoint_rbgs(p, d, 7, 1.4)
        grid.device_status()
        assert (store[1][:s[1]] == 7.0).all() and (store[1][s[1] + n:] == 7.0).all()
        got.append(d.clone())
    assert torch.isfinite(got[0]).all() and torch.equal(got[0], got[1])
    grid.close()


def test_adjoint_rbgs_takes_one_array_of_scratch(dev):
    """hns_adjoint_rbgs alone, launched per colour, allocates a copy of p_bar and no block for the other
    adjoints (two of 2 MiB granules and the tables besides)."""
    from hnanosolver_b200 import lib as hl

    used = []
    for edge in (16, 200):  # the small grid loads the kernels
        grid = hl.Grid(synth.sort_leaves_nanovdb(synth._box_leaves(edge)), voxel_size=0.1)
        grid.set_option(hl.OPT_SPLIT_SOLVE, hl.SPLIT_PER_COLOUR)
        p_bar, d = torch.randn(grid.num_voxels, device=dev), torch.zeros(grid.num_voxels, device=dev)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info(dev)[0]
        grid.adjoint_rbgs(p_bar, d, 4, 1.4)
        grid.device_status()
        used.append(before - torch.cuda.mem_get_info(dev)[0])
        n = grid.num_voxels
        grid.close()
    assert used[1] <= 4 * n + (8 << 20)


@pytest.mark.parametrize("name,floats", [("project", 3), ("confinement", 6)])
def test_adjoints_alone_take_their_own_scratch(dev, name, floats):
    """The adjoint of a projection or of the confinement alone allocates its arrays, not the block of eight
    floats a voxel that the advections' records need (8 MiB of granules and tables besides)."""
    from hnanosolver_b200 import lib as hl

    used = []
    for edge in (16, 200):  # the small grid loads the kernels
        grid = hl.Grid(synth.sort_leaves_nanovdb(synth._box_leaves(edge)), voxel_size=0.1)
        n = grid.num_voxels
        vel, bar, out = (torch.randn((n, 3), device=dev) for _ in range(3))
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info(dev)[0]
        if name == "project":
            grid.adjoint_project(bar, 4, 1.4)
        else:
            grid.adjoint_vorticity_confinement(vel, bar, out, 0.1, 0.4, 1.0)
        grid.device_status()
        used.append(before - torch.cuda.mem_get_info(dev)[0])
        grid.close()
    assert used[1] <= 4 * floats * n + (8 << 20)

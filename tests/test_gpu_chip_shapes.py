"""The solve held in the SMs' shared memory, by shape: how many leaves a CTA holds (four CTAs an SM), so
that neighbours lie in the same CTA as well as in others and the last CTA is short; the CTAs of 256 and
1,024 threads of the transposed sweeps; the sizes at which launches per colour take over. Against one
launch per half-sweep, to the bit. Each case checks by the count of launches which form ran, so that
a grid that took the other form does not pass as compared."""
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


def _leaves(dev, size):
    """A size in leaves: a number, or (k, d) for k leaves per SM and d more."""
    if isinstance(size, int):
        return size
    return size[0] * torch.cuda.get_device_properties(dev).multi_processor_count + size[1]


def _origins(count, shuffled):
    edge = 8 * int(np.ceil(count ** (1.0 / 3.0) + 1e-9))
    o = np.ascontiguousarray(synth.sort_leaves_nanovdb(synth._box_leaves(edge))[:count])
    assert len(o) == count
    return np.ascontiguousarray(np.random.default_rng(0).permutation(o)) if shuffled else o


def _pair(dev, size, shuffled):
    from hnanosolver_b200 import lib as hl

    o = _origins(_leaves(dev, size), shuffled)
    a, b = (hl.Grid(o, voxel_size=0.1) for _ in range(2))
    a.set_option(hl.OPT_SPLIT_SOLVE, hl.SPLIT_AUTO)
    b.set_option(hl.OPT_SPLIT_SOLVE, hl.SPLIT_PER_COLOUR)
    return hl, a, b


def _field(n, dev, seed, comps=1):
    g = torch.Generator(device=dev).manual_seed(seed)
    return torch.randn((n, comps) if comps > 1 else n, device=dev, generator=g)


def _launches(grid, call):
    """The library's launches in one call, a first one (tables, scratch) left out."""
    call()
    grid.device_status()
    grid.profile_read()
    call()
    grid.device_status()
    return grid.profile_read().kernel_launches


@pytest.mark.parametrize("walls", [False, True])
@pytest.mark.parametrize("size,shuffled,held", [((4, 1), False, True), (1300, True, True), (1300, False, True),
                                                (2300, False, True), ((16, 0), True, True), ((16, 1), False, False),
                                                (4096, False, False)])
def test_plain_solve(dev, size, shuffled, held, walls):
    hl, a, b = _pair(dev, size, shuffled)
    n = a.num_voxels
    div, p0 = _field(n, dev, 1), _field(n, dev, 2)
    flags = hl.SOLVE_NEUMANN if walls else 0
    for iterations, extra in ((13, hl.SOLVE_ZERO_INIT), (8, 0)):
        got = []
        for g in (a, b):
            p = p0.clone()

            def solve():
                p.copy_(p0)
                torch.cuda.synchronize()
                g.rbgs(div, p, iterations, 1.6, flags | extra)

            count = _launches(g, solve)
            assert (count == 1) if g is a and held else (count >= 2 * iterations)
            got.append(p)
        assert torch.isfinite(got[0]).all() and torch.equal(got[0], got[1])
    a.close(), b.close()


@pytest.mark.parametrize("walls", [False, True])
@pytest.mark.parametrize("size,shuffled,held", [((4, 1), True, True), ((5, 0), False, True), ((5, 1), False, False)])
def test_checked_solve(dev, size, shuffled, held, walls):
    hl, a, b = _pair(dev, size, shuffled)
    vel = _field(a.num_voxels, dev, 3, 3)
    desc = hl.StepDesc(dt=0.05, max_iterations=46, omega=1.7, tolerance=1e-9, check_every=10,
                       flags=hl.SOLVE_NEUMANN if walls else 0)
    got = []
    for g in (a, b):
        out = torch.empty_like(vel)
        torch.cuda.synchronize()
        g.step_plain(vel, out, [], [], desc)
        solve = g.last_solve()
        g.device_status()
        got.append((out, solve.iterations, solve.residual))
    assert torch.isfinite(got[0][0]).all() and torch.equal(got[0][0], got[1][0]) and got[0][1] == got[1][1] == 46
    # FP64 sums of at most 400,000 terms of one sign in any order: 400,000 x 2^-53 apart.
    assert abs(got[0][2] - got[1][2]) <= 5e-11 * got[1][2]
    # Which form ran: a wait that accepts no face ends only the solve in shared memory.
    a.set_option(hl.OPT_WAIT_POLLS, 0)
    a.step_plain(vel, torch.empty_like(vel), [], [], desc)
    assert hl.lib.hns_device_status(a.handle) == (8 if held else 0)
    a.close(), b.close()


@pytest.mark.parametrize("size,shuffled,held", [((4, 1), False, True), (1300, True, True), ((12, 0), False, True),
                                                ((12, 1), False, False)])
def test_half_precision_inner_solve(dev, size, shuffled, held):
    hl, a, b = _pair(dev, size, shuffled)
    n = a.num_voxels
    vel, dens = _field(n, dev, 4, 3).bfloat16(), _field(n, dev, 5).half()
    desc = hl.MixedDesc(dt=0.05, omega=1.6, tolerance=1e-12, max_outer=3, inner_iterations=15, flags=0)
    got = []
    for g in (a, b):
        vo, do, p = torch.empty_like(vel), torch.empty_like(dens), torch.empty(n, dtype=torch.float64, device=dev)
        torch.cuda.synchronize()
        count = _launches(g, lambda: g.step_mixed(vel, vo, [dens], [do], desc))
        assert (count < 30) if g is a and held else (count >= 90)
        g.refine_pressure(p)
        g.synchronize()
        got.append((vo, do, p))
    for x, y in zip(*got):
        assert torch.isfinite(x).all() and torch.equal(x, y)
    a.close(), b.close()


@pytest.mark.parametrize("size,shuffled,held", [((4, 1), True, True), (1300, False, True), (2300, True, True),
                                                (4100, False, True), (5300, True, True), (6512, False, True),
                                                (6700, False, True), (8000, False, False)])
def test_transposed_sweeps(dev, size, shuffled, held):
    """Up to 4 leaves a CTA of 128 threads, up to 11 of 256 (6,512 leaves on 148 SMs), then one CTA of
    1,024 an SM (6,700)."""
    hl, a, b = _pair(dev, size, shuffled)
    p_bar, d0 = _field(a.num_voxels, dev, 6), _field(a.num_voxels, dev, 7)
    got = []
    for g in (a, b):
        d = d0.clone()

        def sweeps():
            d.copy_(d0)
            torch.cuda.synchronize()
            g.adjoint_rbgs(p_bar, d, 9, 1.4)

        count = _launches(g, sweeps)
        assert (count == 1) if g is a and held else (count == 18)
        got.append(d)
    assert torch.isfinite(got[0]).all() and torch.equal(got[0], got[1])
    a.close(), b.close()


def test_captured_solve_replayed_between_eager_ones(dev):
    """A captured launch has the same tags at every replay: its face words are cleared before it."""
    hl, a, b = _pair(dev, 1300, True)
    n = a.num_voxels
    divs = [_field(n, dev, s) for s in (1, 2, 3)]
    want = []
    for d in divs:
        p = torch.zeros(n, device=dev)
        torch.cuda.synchronize()
        b.rbgs(d, p, 12, 1.6, hl.SOLVE_ZERO_INIT)
        b.synchronize()
        want.append(p)
    stream = torch.cuda.Stream()
    a.set_stream(stream.cuda_stream)
    with torch.cuda.stream(stream):
        div, p, q = divs[0].clone(), torch.zeros(n, device=dev), torch.zeros(n, device=dev)
        a.rbgs(div, p, 12, 1.6, hl.SOLVE_ZERO_INIT)  # makes the tables and the scratch
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            a.rbgs(div, p, 12, 1.6, hl.SOLVE_ZERO_INIT)
        for k in (1, 2, 0, 1):
            div.copy_(divs[k])
            p.zero_()
            graph.replay()
            a.rbgs(divs[2], q, 12, 1.6, hl.SOLVE_ZERO_INIT)
            stream.synchronize()
            a.device_status()
            assert torch.equal(p, want[k]) and torch.equal(q, want[2])
    del graph
    a.close(), b.close()


def test_two_contexts_on_two_streams(dev):
    hl, a, b = _pair(dev, 1300, False)
    c, d = _pair(dev, 700, True)[1:]
    grids = [(a, b, _field(a.num_voxels, dev, 1)), (c, d, _field(c.num_voxels, dev, 2))]
    outs = [[torch.zeros_like(div) for _ in range(12)] for _, _, div in grids]
    torch.cuda.synchronize()
    for k in range(12):
        for (g, _, div), out in zip(grids, outs):
            g.rbgs(div, out[k], 8 + k, 1.6, hl.SOLVE_ZERO_INIT)
    for g, ref, div in grids:
        g.device_status()
    for (g, ref, div), out in zip(grids, outs):
        for k in range(12):
            p = torch.zeros_like(div)
            torch.cuda.synchronize()
            ref.rbgs(div, p, 8 + k, 1.6, hl.SOLVE_ZERO_INIT)
            ref.synchronize()
            assert torch.equal(out[k], p)
    for g in (a, b, c, d):
        g.close()

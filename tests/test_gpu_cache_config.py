"""A program that prefers L1 over shared memory (cuCtxSetCacheConfig, cudaDeviceSetCacheConfig), from the
start or from some call on: the solves that would be held in shared memory run, with the same values. Their
CTAs must all be resident at once, and the preference leaves room for one an SM."""
import ctypes

import numpy as np
import pytest

from hnanosolver_b200 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

PREFER = {"shared": 1, "L1": 2, "equal": 3}


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda", 0)


@pytest.mark.parametrize("leaves", [592, 2368, 4100, 6512, 6700])
@pytest.mark.parametrize("prefer", sorted(PREFER))
def test_solves_launch_under_any_preference(dev, prefer, leaves):
    from hnanosolver_b200 import lib as hl

    driver = ctypes.CDLL("libcuda.so.1")
    edge = 8 * int(np.ceil(leaves ** (1.0 / 3.0)))
    grid = hl.Grid(np.ascontiguousarray(synth.sort_leaves_nanovdb(synth._box_leaves(edge))[:leaves]), voxel_size=0.1)
    gen = torch.Generator(device=dev).manual_seed(3)
    div = torch.randn(grid.num_voxels, device=dev, generator=gen)
    got = []
    try:
        for config in (PREFER[prefer], 0, PREFER[prefer]):
            assert driver.cuCtxSetCacheConfig(config) == 0
            p, w, d = (torch.zeros_like(div) for _ in range(3))
            torch.cuda.synchronize()
            grid.rbgs(div, p, 9, 1.5, hl.SOLVE_ZERO_INIT)
            grid.rbgs(div, w, 9, 1.5, hl.SOLVE_ZERO_INIT | hl.SOLVE_NEUMANN)
            grid.adjoint_rbgs(div, d, 9, 1.5)
            grid.device_status()
            got.append((p, w, d))
    finally:
        driver.cuCtxSetCacheConfig(0)
    for a, b, c in zip(*got):
        assert torch.isfinite(a).all() and torch.equal(a, b) and torch.equal(a, c)
    grid.close()

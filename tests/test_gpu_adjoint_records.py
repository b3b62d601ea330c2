"""The reverse pass of the step's advections as one launch for the velocity and all scalars, against
the same adjoints taken one field at a time: 0, 1, 3 and 17 scalars (more than one launch carries),
traces of up to several voxels that leave the domain. Both sum the same terms in FP32 in another
order; a voxel receives at most a few hundred of them, so they agree to 1e-5 of the largest value."""
import numpy as np
import pytest

from hnanosolver_b200 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nscalars,speed", [(0, 1.0), (1, 1.0), (3, 6.0), (17, 1.0)])
def test_step_adjoint_is_the_sum_of_its_fields(nscalars, speed):
    from hnanosolver_b200 import lib as hl

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    dev = torch.device("cuda", 0)
    origins = synth.spheres_topology(64, 2, 8.0, 16.0, seed=3)
    _, vel = synth.smoothed_fields(origins, seed=0, box_passes=1)
    g = hl.Grid(origins, voxel_size=0.1)
    v = torch.from_numpy(np.ascontiguousarray(vel * speed)).to(dev)
    rng = torch.Generator(device=dev).manual_seed(1)
    rand = lambda *s: torch.randn(s, device=dev, generator=rng)  # noqa: E731
    n = g.num_voxels
    scalars, bars = [rand(n) for _ in range(nscalars)], [rand(n) for _ in range(nscalars)]
    vel_bar = rand(n, 3)
    got_v, got = torch.zeros_like(v), [torch.zeros(n, device=dev) for _ in range(nscalars)]
    ref_v, ref = torch.zeros_like(v), [torch.zeros(n, device=dev) for _ in range(nscalars)]
    projected = vel_bar.clone()
    torch.cuda.synchronize()
    g.adjoint_step_plain(v, scalars, vel_bar, bars, got_v, got, 0.1, 5, 1.2)
    g.adjoint_project(projected, 5, 1.2)
    g.adjoint_advect_vec3(v, projected, ref_v, 0.1)
    for d, b, r in zip(scalars, bars, ref):
        g.adjoint_advect_scalar(v, d, b, r, ref_v, 0.1)
    g.synchronize()
    for x, y in zip([got_v, *got], [ref_v, *ref]):
        assert float((x - y).abs().max()) <= 1e-5 * float(y.abs().max())
    g.close()

"""The column transforms of the phi precompute at every size, in both bases, on both sides of the grid split."""
import numpy as np
import pytest

from conftest import rel_l2
from oracle import lenseflow_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,B", [(64, 30), (128, 17), (256, 9), (512, 5), (1024, 2)])
def test_planes_do_not_depend_on_the_batch_and_lens_matches_oracle(N, B):
    """A batch takes one block per column tile, a map alone three: the same bits, derivative planes and p planes, for
    a MAP and a FOURIER phi; and the float64 lens that reads the planes matches the oracle to the engine's 1e-10."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cmblensing_b200 import engine
    from cmblensing_b200.simulate import lens_batch
    theta, n = (3.0 if N <= 256 else 2.0), 2
    pw = R.pix_width_of(theta)
    f, two = lens_batch(N, theta, 2, 1, seed0=150)
    plan = engine.get_plan(N, 1, pw, "f64")
    p32 = engine.get_plan(N, 1, pw)
    for given in (two, np.fft.rfft2(two)):
        phi = torch.as_tensor(given, device="cuda")[[i % 2 for i in range(B)]].contiguous()
        planes = plan.phi_planes(phi)
        pp = p32.phi_pp(phi, n)
        assert all(v > 0.0 for v in p32.last_min_det)
        for i in (0, B - 1):
            alone = plan.phi_planes(phi[i:i + 1])
            assert torch.equal(alone[0], planes[i])
            assert torch.equal(p32.phi_pp(phi[i:i + 1], n)[0], pp[i])
        k = (B - 1) % 2
        got = plan.lense_flow(torch.as_tensor(f[k:k + 1], device="cuda"), alone, n=n)[0, 0].cpu().numpy()
        assert rel_l2(got, R.primal_lense_flow(f[k, 0], given[k], pw, n, 1, False)) < 1e-10

"""The stage-time p planes, p = M(t)^-1 grad(phi), to the last bit that their arithmetic has."""
import numpy as np
import pytest

from oracle import lenseflow_ref as R

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("N", [64, 512])
def test_from_derivative_planes(torch_cuda, N):
    """float64 arithmetic and one rounding to float32, with the reference's det + 1e-12, also where M is singular or
    nearly so: phi_xx = -1 + 2^-j and -1 itself, at quarter times, where numpy's float64 formula is exact up to the
    1e-12 and the quotient.  Tolerance: half a float32 unit (2^-24), and 2^-44 for both sides' float64 roundings."""
    torch = torch_cuda
    from cmblensing_b200 import engine
    n = 2
    plan = engine.get_plan(N, 1, R.pix_width_of(2.0))
    rng = np.random.default_rng(5)
    d = np.zeros((5, N, N), dtype=np.float32)
    d[0], d[1] = rng.uniform(0.5, 2.0, (2, N, N))
    j = rng.integers(0, 25, (N, N))
    d[2] = np.where(j == 24, -1.0, -1.0 + 2.0 ** -np.minimum(j, 23)).astype(np.float32)
    d[2, 0] = -1.0
    f = torch.zeros((1, 1, N, N), dtype=torch.float32, device="cuda")
    base = plan.workspace_bytes(1, False)
    ws = torch.empty(plan.workspace_bytes(1, False, n), dtype=torch.uint8, device="cuda")
    plan.lense_flow(f, torch.as_tensor(d[None], device="cuda"), n=n, workspace=ws)
    pp = ws[base:].view(torch.float32).view(2 * n + 1, 2, N, N).cpu().numpy()
    px, py, pxx = (d[k].astype(np.float64) for k in range(3))
    for k in range(2 * n + 1):
        m = 1.0 + k / (2.0 * n) * pxx
        for got, want in ((pp[k, 0], px / (m + 1e-12)), (pp[k, 1], py * m / (m + 1e-12))):
            err = np.abs(got - want)
            assert np.all(err <= (2.0 ** -24 + 2.0 ** -44) * np.abs(want) + 2.0 ** -50), (k, np.max(err / np.abs(want)))

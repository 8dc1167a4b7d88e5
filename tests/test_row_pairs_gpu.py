"""The row-pair passes (512^2 with one or three components, 1024^2) against the general row pass and the oracle."""
import pytest

from conftest import rel_l2
from oracle import lenseflow_ref as R

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("N,C,B,n", [(512, 1, 3, 2), (512, 3, 1, 1), (1024, 1, 2, 1), (1024, 2, 1, 3), (1024, 3, 1, 2)])
@pytest.mark.parametrize("adjoint", [False, True])
def test_row_pairs_match_general_pass_and_oracle(torch_cuda, N, C, B, n, adjoint):
    """The p-plane path (row pairs) and the derivative-plane path (general row pass) against the oracle to 1e-5;
    batch and alone bit for bit.  (The two differ by more than rounding here: at two-arcminute pixels one to
    three RK4 steps are below the scheme's stability limit and amplify the rounding of the highest modes.)"""
    torch = torch_cuda
    from cmblensing_b200 import engine
    from cmblensing_b200.simulate import lens_batch
    theta = 2.0
    f, phis = lens_batch(N, theta, B, C, seed0=130)
    pw = R.pix_width_of(theta)
    plan = engine.get_plan(N, C, pw)
    planes = plan.phi_planes(torch.as_tensor(phis, device="cuda"))
    ft = torch.as_tensor(f, device="cuda", dtype=torch.float32)
    outs = []
    for nbytes in (plan.workspace_bytes(B, adjoint), plan.workspace_bytes(B, adjoint, n)):
        ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        outs.append(plan.lense_flow(ft, planes, n=n, direction=-1, adjoint=adjoint, workspace=ws))
    ref = R.primal_lense_flow(f[B - 1, C - 1], phis[B - 1], pw, n, -1, adjoint)
    for out in outs:
        assert rel_l2(out[B - 1, C - 1].double().cpu().numpy(), ref) < 1e-5
    one = plan.lense_flow(ft[B - 1:], planes[B - 1:], n=n, direction=-1, adjoint=adjoint)
    assert torch.equal(one[0], outs[1][B - 1])
    assert engine.wait_timeouts() == 0

"""Every map and component of a batch, and the field types, on the routes that the other tests sample."""
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


@pytest.mark.parametrize("N,C,B", [(512, 1, 2), (512, 3, 2), (1024, 2, 1), (1024, 3, 1)])
@pytest.mark.parametrize("adjoint", [False, True])
def test_row_pairs(torch_cuda, N, C, B, adjoint):
    """The row-pair passes against the oracle, to the engine's 1e-5; float64 fields in, lensed in place and out of
    place, have the bits of float32 fields in (the same values) to a rounding of the output."""
    torch = torch_cuda
    from cmblensing_b200 import engine
    from cmblensing_b200.simulate import lens_batch
    theta, n = 2.0, 2
    f, phis = lens_batch(N, theta, B, C, seed0=270)
    pw = R.pix_width_of(theta)
    plan = engine.get_plan(N, C, pw)
    planes = plan.phi_planes(torch.as_tensor(phis, device="cuda"))
    f32 = torch.as_tensor(f, device="cuda", dtype=torch.float32)
    got = plan.lense_flow(f32, planes, n=n, adjoint=adjoint)
    f = f32.double().cpu().numpy()
    for b in range(B):
        for c in range(C):
            ref = R.primal_lense_flow(f[b, c], phis[b], pw, n, 1, adjoint)
            assert rel_l2(got[b, c].double().cpu().numpy(), ref) < 1e-5, (b, c)
    f64 = f32.double()
    wide = plan.lense_flow(f64, planes, n=n, adjoint=adjoint)
    assert wide.dtype == torch.float64 and torch.equal(wide.float(), got) and torch.equal(wide, got.double())
    assert torch.equal(plan.lense_flow(f64, planes, n=n, adjoint=adjoint, out=f64), wide)
    assert torch.equal(plan.lense_flow(f32, planes, n=n, adjoint=adjoint, out=f32), got)


@pytest.mark.parametrize("N", [64, 128, 256])
@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("n,direction", [(1, 1), (3, -1)])
def test_float64_clusters_with_p_planes(torch_cuda, N, adjoint, n, direction):
    """The default route of a float64 lens: every map and component against the oracle to 1e-10, and the route that forms
    p in the kernel (whose stage times may differ in their last bit) to 1e-13."""
    torch = torch_cuda
    from cmblensing_b200 import engine
    from cmblensing_b200.simulate import lens_batch
    B, C, theta = 3, 2, 3.0
    f, phis = lens_batch(N, theta, B, C, seed0=290)
    pw = R.pix_width_of(theta)
    plan = engine.get_plan(N, C, pw, "f64")
    planes = plan.phi_planes(torch.as_tensor(phis, device="cuda"))
    ft = torch.as_tensor(f, device="cuda")
    got = plan.lense_flow(ft, planes, n=n, direction=direction, adjoint=adjoint).cpu().numpy()
    small = torch.empty(plan.workspace_bytes(B, adjoint), dtype=torch.uint8, device="cuda")
    other = plan.lense_flow(ft, planes, n=n, direction=direction, adjoint=adjoint, workspace=small).cpu().numpy()
    for b in range(B):
        for c in range(C):
            ref = R.primal_lense_flow(f[b, c], phis[b], pw, n, direction, adjoint)
            assert rel_l2(got[b, c], ref) < 1e-10, (b, c)
    assert rel_l2(other, got) < 1e-13

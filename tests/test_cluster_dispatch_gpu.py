"""256^2 lenses of two and three components without room for all p planes: step by step, with the bits of the lens
that has them."""
import pytest

from oracle import lenseflow_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,B", [(2, 1), (2, 15), (3, 5), (3, 29)])
@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("adjoint,direction", [(False, 1), (False, -1), (True, 1), (True, -1)])
@pytest.mark.parametrize("n", [1, 3, 7])
def test_steps_have_the_bits_of_the_whole_lens(C, B, prec, adjoint, direction, n):
    """Few maps and more than fit on the GPU at once; all directions of time; fields of either type in and out, and a
    single step in place between types."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cmblensing_b200 import engine
    from cmblensing_b200.simulate import lens_batch
    N = 256
    f, phis = lens_batch(N, 3.0, 2, C, seed0=250)
    reps = [i % 2 for i in range(B)]
    plan = engine.get_plan(N, C, R.pix_width_of(3.0), prec)
    planes = plan.phi_planes(torch.as_tensor(phis, device="cuda")[reps].contiguous())
    f = torch.as_tensor(f, device="cuda")[reps].contiguous()
    ws = torch.empty(plan.workspace_bytes(B, adjoint), dtype=torch.uint8, device="cuda")
    full = torch.empty(plan.workspace_bytes(B, adjoint, n), dtype=torch.uint8, device="cuda")
    for tin, tout in ((torch.float32, torch.float32), (torch.float64, torch.float32), (torch.float32, torch.float64)):
        x = f.to(tin)
        got = plan.lense_flow(x, planes, n=n, direction=direction, adjoint=adjoint, workspace=ws, out_dtype=tout)
        want = plan.lense_flow(x, planes, n=n, direction=direction, adjoint=adjoint, workspace=full, out_dtype=tout)
        assert torch.equal(got, want)
    raw = torch.empty(8 * f.numel(), dtype=torch.uint8, device="cuda")
    fi = raw[:4 * f.numel()].view(torch.float32).view(f.shape)
    fo = raw.view(torch.float64).view(f.shape)
    fi.copy_(f)
    plan.lense_flow(fi, planes, n=n, direction=direction, adjoint=adjoint, workspace=ws, out=fo)
    assert torch.equal(fo, want)
    assert engine.wait_timeouts() == 0

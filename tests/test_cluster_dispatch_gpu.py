"""Both sides of the lines between the cluster kernels and the row and column passes at 256^2: the route that is taken
and the same fields."""
import pytest

from conftest import rel_l2
from oracle import lenseflow_ref as R

pytestmark = pytest.mark.gpu


def _problem(torch, C, B, prec):
    from cmblensing_b200 import engine
    from cmblensing_b200.simulate import lens_batch
    N = 256
    f, phis = lens_batch(N, 3.0, 2, C, seed0=250)
    reps = [i % 2 for i in range(B)]
    plan = engine.get_plan(N, C, R.pix_width_of(3.0), prec)
    ft = torch.as_tensor(f, device="cuda", dtype=plan.dtype)[reps].contiguous()
    return plan, ft, plan.phi_planes(torch.as_tensor(phis, device="cuda")[reps].contiguous())


def _columns(plan, run):
    """Column passes that run() launched."""
    from cmblensing_b200 import _native as nat
    plan.profile()
    try:
        out = run()
        return out, plan.profile_read(nat.LF_KIND_COL)[1]
    finally:
        plan.profile(False)
        plan.profile_reset()


@pytest.mark.parametrize("C,B,adjoint,passes", [(2, 14, False, False), (2, 15, False, True), (2, 28, True, False),
                                                (2, 29, True, True), (3, 20, False, False), (1, 40, False, False)])
def test_lens_without_p_planes(C, B, adjoint, passes):
    """14 clusters at once: QU lenses change over above two (adjoint four) times as many component planes.  Against the
    p-plane path: two roundings of about 1e-7, bound 1e-6."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n = 3
    plan, f, planes = _problem(torch, C, B, "f32")
    ws = torch.empty(plan.workspace_bytes(B, adjoint), dtype=torch.uint8, device="cuda")
    got, columns = _columns(plan, lambda: plan.lense_flow(f, planes, n=n, adjoint=adjoint, workspace=ws))
    assert columns == (4 * n if passes else 0)
    want, columns = _columns(plan, lambda: plan.lense_flow(f, planes, n=n, adjoint=adjoint))
    assert columns == 0
    assert rel_l2(got.cpu().numpy(), want.cpu().numpy()) < 1e-6


@pytest.mark.parametrize("C,B,passes", [(2, 42, False), (2, 43, True), (3, 18, False), (3, 19, True), (1, 64, False)])
def test_float64_reverse_pass(C, B, passes):
    """Seven clusters at once: above 84 planes of QU maps and 56 of TQU maps.  Each map against a batch of two, which
    runs on clusters, to the float64 engine's 1e-10."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n = 1
    plan, f, planes = _problem(torch, C, B, "f64")
    cot = f.flip(-1).contiguous()
    got, columns = _columns(plan, lambda: plan.lense_flow_vjp(f, cot, planes, n=n, return_f=True))
    assert columns == (2 * 4 * n if passes else 0)
    want, columns = _columns(plan, lambda: plan.lense_flow_vjp(f[:2], cot[:2], planes[:2], n=n, return_f=True))
    assert columns == 0
    for a, b in zip(got, want):
        for i in (0, 1, B - 1):
            assert rel_l2(a[i].cpu().numpy(), b[i % 2].cpu().numpy()) < 1e-10

"""The cluster-resident lens (N <= 256: one launch integrates every component map) against the float64 oracle.

Tolerances: those of the engine, relative L2 1e-5 for float32 compute and 1e-10 for float64.
"""
import numpy as np
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


@pytest.mark.parametrize("N", [64, 128, 256])
@pytest.mark.parametrize("prec,planes", [("f32", "p"), ("f32", "derivatives"), ("f64", "derivatives")])
@pytest.mark.parametrize("adjoint", [False, True])
def test_every_kernel_matches_oracle(torch_cuda, N, prec, planes, adjoint):
    """Each instantiation (size, precision, p source, right-hand side) on an odd batch of two-component maps,
    one RK4 step and three, both directions; the p planes and the derivative planes are selected by the
    workspace size as in lf_lense_flow."""
    torch = torch_cuda
    from cmblensing_b200 import engine
    from cmblensing_b200.simulate import lens_batch
    B, C, theta = 3, 2, 3.0
    f, phis = lens_batch(N, theta, B, C, seed0=70)
    pw = R.pix_width_of(theta)
    plan = engine.get_plan(N, C, pw, prec)
    pl = plan.phi_planes(torch.as_tensor(phis, device="cuda"))
    ft = torch.as_tensor(f, device="cuda", dtype=plan.dtype)
    for n, direction in ((1, 1), (3, -1)):
        nbytes = plan.workspace_bytes(B, adjoint, n if planes == "p" else None)
        ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        got = plan.lense_flow(ft, pl, n=n, direction=direction, adjoint=adjoint, workspace=ws).double().cpu().numpy()
        for b in (0, B - 1):
            for c in range(C):
                ref = R.primal_lense_flow(f[b, c], phis[b], pw, n, direction, adjoint)
                assert rel_l2(got[b, c], ref) < (1e-10 if prec == "f64" else 1e-5), (n, direction, b, c)


@pytest.mark.parametrize("N,B", [(64, 41), (128, 23), (256, 9)])
def test_more_clusters_than_fit_and_two_streams(torch_cuda, N, B):
    """More component maps than clusters fit on the GPU, on two streams at once: every map equals the same map
    lensed alone, bit for bit."""
    torch = torch_cuda
    from cmblensing_b200 import engine
    from cmblensing_b200.simulate import lens_batch
    C, n = 3, 2
    f, phis = lens_batch(N, 3.0, 4, C, seed0=90)
    reps = [i % 4 for i in range(B)]
    plan = engine.get_plan(N, C, R.pix_width_of(3.0))
    ft = torch.as_tensor(f, device="cuda", dtype=torch.float32)[reps].contiguous()
    pp = plan.phi_pp(torch.as_tensor(phis, device="cuda"), n)[reps].contiguous()
    alone = [plan.lense_flow_pp(ft[i:i + 1], pp[i:i + 1], n) for i in range(4)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    outs = []
    for s in streams:
        with torch.cuda.stream(s):
            outs.append(plan.lense_flow_pp(ft, pp, n))
    torch.cuda.synchronize()
    for out in outs:
        for i in range(B):
            assert torch.equal(out[i], alone[reps[i]][0]), i
    assert engine.wait_timeouts() == 0


def _grad_problem(torch, N, C, B, n):
    from cmblensing_b200 import engine
    from cmblensing_b200.simulate import lens_batch
    f, phis = lens_batch(N, 3.0, B, C, seed0=110)
    pw = R.pix_width_of(3.0)
    cot = np.random.default_rng(111).standard_normal(f.shape)
    out = {}
    for prec in ("f32", "f64"):
        plan = engine.get_plan(N, C, pw, prec)
        planes = plan.phi_planes(torch.as_tensor(phis, device="cuda"))
        out[prec] = (plan, planes, torch.as_tensor(f, device="cuda", dtype=plan.dtype),
                     torch.as_tensor(cot, device="cuda", dtype=plan.dtype))
    return out


@pytest.mark.parametrize("N,C,n", [(64, 1, 1), (64, 3, 2), (128, 2, 1), (128, 1, 14), (256, 3, 1), (256, 2, 3)])
@pytest.mark.parametrize("scheme", ["reference", "exact"])
def test_reverse_passes_float32_against_float64(torch_cuda, N, C, n, scheme):
    """Both reverse schemes, one launch pair per RK4 step, at the edges of their step counts (a single step; more
    steps than the forward lens's p planes find room for): float32 within the engine's gradient tolerance 2e-5 of
    the float64 engine, which the oracle pins (test_vjp_gpu)."""
    torch = torch_cuda
    got = {}
    for prec, (plan, planes, f, cot) in _grad_problem(torch, N, C, 2, n).items():
        fn = plan.lense_flow_vjp_ckpt if scheme == "exact" else plan.lense_flow_vjp
        got[prec] = [x.cpu().numpy() for x in fn(f, cot, planes, n, phi_basis="map")] + \
                    [x.cpu().numpy() for x in fn(f, cot, planes, n, -1, "fourier", True)]
    for a, b in zip(got["f32"], got["f64"]):
        assert rel_l2(a, b) < 2e-5


def test_single_step_reverse_pass_in_place(torch_cuda):
    """A one-step reverse pass whose delta-f overwrites the lensed field it reads: as with separate buffers."""
    import ctypes
    torch = torch_cuda
    from cmblensing_b200 import _native as nat
    N, C, B = 64, 2, 5
    plan, planes, f, cot = _grad_problem(torch, N, C, B, 1)["f32"]
    df, dphi = plan.lense_flow_vjp(f, cot, planes, 1)
    g = f.clone()
    dphi2 = torch.empty_like(dphi)
    nbytes = plan._lib.lf_vjp_workspace_bytes(plan.handle, B)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    nat.check(plan._lib.lf_lense_flow_vjp(plan.handle, ptr(g), ptr(cot), nat.LF_F32, ptr(planes), B, 1, 1, ptr(g), None,
                                          ptr(dphi2), nat.LF_PHI_FOURIER, ptr(ws), nbytes,
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    assert torch.equal(g, df) and torch.equal(dphi2, dphi)

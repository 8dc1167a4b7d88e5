"""Calls whose output shares memory with their inputs, where the lens runs plane by plane (N <= 256): the same bits as
with separate buffers."""
import ctypes

import pytest

from oracle import lenseflow_ref as R

pytestmark = pytest.mark.gpu

# more component maps than clusters fit on the GPU at once
SIZES = [(64, 90), (128, 41), (256, 9)]


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _problem(torch, N, B, C, prec="f32"):
    from cmblensing_b200 import engine
    from cmblensing_b200.simulate import lens_batch
    f, phis = lens_batch(N, 3.0, 3, C, seed0=170)
    plan = engine.get_plan(N, C, R.pix_width_of(3.0), prec)
    reps = [i % 3 for i in range(B)]
    scale = torch.arange(1, B + 1, device="cuda", dtype=torch.float64).view(B, 1, 1, 1)  # every map another one
    ft = torch.as_tensor(f, device="cuda")[reps] * scale / B
    return plan, ft.contiguous(), torch.as_tensor(phis, device="cuda")[reps].contiguous()


@pytest.mark.parametrize("N,B", SIZES)
@pytest.mark.parametrize("prec,path", [("f32", "p"), ("f32", "derivatives"), ("f32", "given p"), ("f64", "p")])
@pytest.mark.parametrize("narrowing", [False, True])
def test_lens_in_place_between_types(torch_cuda, N, B, prec, path, narrowing):
    """float32 in and float64 out (and the reverse) from one address: an early plane's output covers other planes'
    input."""
    torch = torch_cuda
    C, n = 3, 2
    plan, f, phi = _problem(torch, N, B, C, prec)
    tin, tout = (torch.float64, torch.float32) if narrowing else (torch.float32, torch.float64)
    f = f.to(tin)
    raw = torch.empty(8 * f.numel(), dtype=torch.uint8, device="cuda")
    fi = raw[:f.numel() * f.element_size()].view(tin).view(f.shape)
    fo = raw[:f.numel() * (4 if narrowing else 8)].view(tout).view(f.shape)
    if path == "given p":
        pp = plan.phi_pp(phi, n)
        lens = lambda x, y: plan.lense_flow_pp(x, pp, n, out=y)
    else:
        planes = plan.phi_planes(phi)
        ws = torch.empty(plan.workspace_bytes(B, False, n if path == "p" else None), dtype=torch.uint8, device="cuda")
        lens = lambda x, y: plan.lense_flow(x, planes, n=n, out=y, workspace=ws)
    want = lens(f, torch.empty(f.shape, dtype=tout, device="cuda"))
    for _ in range(3):  # (which clusters come first may differ)
        fi.copy_(f)
        assert lens(fi, fo).data_ptr() == fi.data_ptr()
        assert torch.equal(fo, want)


@pytest.mark.parametrize("N,B", SIZES)
def test_lens_into_shifted_input_and_into_its_planes(torch_cuda, N, B):
    """An output one map behind the input, and one over the derivative planes that the lens reads."""
    torch = torch_cuda
    C, n = 3, 2
    plan, f, phi = _problem(torch, N, B, C)
    f = f.float()
    planes = plan.phi_planes(phi)
    ws = torch.empty(plan.workspace_bytes(B, True), dtype=torch.uint8, device="cuda")
    want = plan.lense_flow(f, planes, n=n, adjoint=True, workspace=ws)
    buf = torch.empty((B + 1, C, N, N), dtype=torch.float32, device="cuda")
    buf[:B] = f
    got = plan.lense_flow(buf[:B], planes, n=n, adjoint=True, out=buf[1:], workspace=ws)
    assert torch.equal(got, want)
    over = planes.view(-1)[:f.numel()].view(f.shape)
    plan.lense_flow(f, planes, n=n, adjoint=True, out=over, workspace=ws)
    assert torch.equal(over, want)


def test_noalloc_in_place_between_types(torch_cuda):
    """The allocation-free entry point at a batch near its scratch limit."""
    torch = torch_cuda
    from cmblensing_b200 import _native as nat
    N, B, C, n = 64, 120, 3, 2
    plan, f, phi = _problem(torch, N, B, C)
    planes = plan.phi_planes(phi)
    raw = f.clone()
    out = raw.view(-1).view(torch.float32)[:f.numel()].view(f.shape)
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    want = torch.empty(f.shape, dtype=torch.float32, device="cuda")
    for x, y in ((f, want), (raw, out)):
        nat.check(plan._lib.lf_lense_flow_noalloc(N, C, plan.pix_width, ptr(x), nat.LF_F64, ptr(y), nat.LF_F32,
                                                  ptr(planes), B, n, 1, 0, st))
    torch.cuda.synchronize()
    assert torch.equal(out, want)


def _reverse(torch, scheme, plan, B, n, f, cot, planes, out, other, dphi, io):
    """lf_lense_flow_vjp (``other``: the re-integrated field) or lf_lense_flow_vjp_ckpt (``other``: the lensed field)."""
    from cmblensing_b200 import _native as nat
    lib, ptr = plan._lib, lambda t: ctypes.c_void_p(t.data_ptr()) if t is not None else None
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    if scheme == "exact":
        nbytes = lib.lf_vjp_ckpt_workspace_bytes(plan.handle, B, n)
        ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        nat.check(lib.lf_lense_flow_vjp_ckpt(plan.handle, ptr(f), ptr(cot), io, ptr(planes), B, n, 1, ptr(other), ptr(out),
                                             ptr(dphi), nat.LF_PHI_FOURIER, ptr(ws), nbytes, st))
    else:
        nbytes = lib.lf_vjp_workspace_bytes(plan.handle, B)
        ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        nat.check(lib.lf_lense_flow_vjp(plan.handle, ptr(f), ptr(cot), io, ptr(planes), B, n, 1, ptr(out), ptr(other),
                                        ptr(dphi), nat.LF_PHI_FOURIER, ptr(ws), nbytes, st))
    torch.cuda.synchronize()


@pytest.mark.parametrize("N,B", [(64, 90), (256, 7)])
@pytest.mark.parametrize("io64", [False, True])
@pytest.mark.parametrize("case", ["back over cotangent", "swapped", "delta one map on", "delta over planes",
                                  "exact: delta one map on", "exact: delta over planes"])
@pytest.mark.parametrize("n", [1, 2])
def test_reverse_pass_outputs_over_inputs(torch_cuda, N, B, io64, case, n):
    """The two systems of a reverse step run side by side: outputs over the other system's input (a single step reads
    it until its end), over a neighbour's plane, over the derivative planes (read until the last delta-phi terms)."""
    torch = torch_cuda
    from cmblensing_b200 import _native as nat
    C = 2
    scheme = "exact" if case.startswith("exact") else "reference"
    plan, f, phi = _problem(torch, N, B, C)
    dt, io = (torch.float64, nat.LF_F64) if io64 else (torch.float32, nat.LF_F32)
    f = f.to(dt)
    cot = f.flip(0).flip(-1).contiguous()
    planes = plan.phi_planes(phi)
    dphi = torch.empty((B, N, N // 2 + 1), dtype=torch.complex128, device="cuda")
    want, other, want_dphi = torch.empty_like(f), torch.empty_like(f), torch.empty_like(dphi)
    _reverse(torch, scheme, plan, B, n, f, cot, planes, want, other, want_dphi, io)
    fi, ci, pi = f.clone(), cot.clone(), planes.clone()
    out, back = torch.empty_like(f), None
    if case == "back over cotangent":
        back = ci
    elif case == "swapped":
        out, back = fi, ci
    elif case.endswith("one map on"):
        buf = torch.empty((B + 1, C, N, N), dtype=dt, device="cuda")
        buf[:B] = cot
        ci, out = buf[:B], buf[1:]
    else:
        out = pi.view(-1).view(dt)[:f.numel()].view(f.shape)
    _reverse(torch, scheme, plan, B, n, fi, ci, pi, out, back, dphi, io)
    assert torch.equal(out, want) and torch.equal(dphi, want_dphi)
    if back is not None:
        assert torch.equal(back, other)


@pytest.mark.parametrize("n", [3, 9])
def test_checkpointed_pass_with_a_shifted_lensed_field(torch_cuda, n):
    """The lensed field one map behind the input, with step counts whose p planes end before and in the last of the
    workspace's regions that the forward lens may use."""
    torch = torch_cuda
    from cmblensing_b200 import _native as nat
    N, B, C = 256, 20, 2
    plan, f, phi = _problem(torch, N, B, C)
    f = f.float()
    cot = f.flip(0).contiguous()
    planes = plan.phi_planes(phi)
    dphi = torch.empty((B, N, N // 2 + 1), dtype=torch.complex128, device="cuda")
    want, lensed, want_dphi = torch.empty_like(f), torch.empty_like(f), torch.empty_like(dphi)
    _reverse(torch, "exact", plan, B, n, f, cot, planes, want, lensed, want_dphi, nat.LF_F32)
    buf = torch.empty((B + 1, C, N, N), dtype=torch.float32, device="cuda")
    buf[:B] = f
    out = torch.empty_like(f)
    _reverse(torch, "exact", plan, B, n, buf[:B], cot, planes, out, buf[1:], dphi, nat.LF_F32)
    assert torch.equal(buf[1:], lensed) and torch.equal(out, want) and torch.equal(dphi, want_dphi)

"""Streams that may use part of the SMs only (a green context), where clusters have no place: lenses and reverse passes of
N <= 256 run there too, with a launch per stage."""
import ctypes

import pytest

from conftest import rel_l2
from oracle import lenseflow_ref as R

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def small_stream():
    """A stream on 16 SMs that were split off without regard to clusters, so that none fits."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    driver = pytest.importorskip("cuda.bindings.driver")
    torch.cuda.synchronize()

    def ok(r):
        assert r[0] == driver.CUresult.CUDA_SUCCESS, r[0]
        return r[1:]

    dev, = ok(driver.cuDeviceGet(torch.cuda.current_device()))
    whole, = ok(driver.cuDeviceGetDevResource(dev, driver.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    split = driver.CUdevSmResourceSplit_flags.CU_DEV_SM_RESOURCE_SPLIT_IGNORE_SM_COSCHEDULING
    groups, _, _ = ok(driver.cuDevSmResourceSplitByCount(1, whole, split, 16))
    desc, = ok(driver.cuDevResourceGenerateDesc(groups, 1))
    ctx, = ok(driver.cuGreenCtxCreate(desc, dev, driver.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    stream, = ok(driver.cuGreenCtxStreamCreate(ctx, driver.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    yield torch.cuda.ExternalStream(int(stream))
    torch.cuda.synchronize()
    ok(driver.cuStreamDestroy(stream))
    ok(driver.cuGreenCtxDestroy(ctx))


def _problem(torch, N, C, B, prec):
    from cmblensing_b200 import engine
    from cmblensing_b200.simulate import lens_batch
    f, phis = lens_batch(N, 3.0, B, C, seed0=230)
    plan = engine.get_plan(N, C, R.pix_width_of(3.0), prec)
    return plan, torch.as_tensor(f, device="cuda", dtype=plan.dtype), torch.as_tensor(phis, device="cuda")


@pytest.mark.parametrize("N,C", [(64, 1), (128, 3), (256, 2)])
@pytest.mark.parametrize("prec,path", [("f32", "p"), ("f32", "derivatives"), ("f32", "given p"), ("f64", "p")])
@pytest.mark.parametrize("adjoint,direction", [(False, 1), (True, 1), (False, -1)])
def test_lens(small_stream, N, C, prec, path, adjoint, direction):
    """Against the same lens on the whole GPU: two roundings of about 1e-7 in float32 (bound 1e-6), 1e-10 in float64; as
    many column passes as stages."""
    import torch
    from cmblensing_b200 import _native as nat
    B, n = 3, 4
    plan, f, phi = _problem(torch, N, C, B, prec)
    planes = plan.phi_planes(phi)
    ws = torch.empty(plan.workspace_bytes(B, adjoint, None if path == "derivatives" else n), dtype=torch.uint8,
                     device="cuda")
    outs = [torch.empty_like(f), torch.empty_like(f)]
    if path == "given p":
        pp = plan.phi_pp(phi, n)
        lens = lambda out: plan.lense_flow_pp(f, pp, n, direction, adjoint, out=out, workspace=ws)
    else:
        lens = lambda out: plan.lense_flow(f, planes, n, direction, adjoint, out=out, workspace=ws)
    lens(outs[0])
    torch.cuda.synchronize()
    plan.profile()
    try:
        with torch.cuda.stream(small_stream):
            lens(outs[1])
        small_stream.synchronize()
        assert plan.profile_read(nat.LF_KIND_COL)[1] == 4 * n
    finally:
        plan.profile(False)
        plan.profile_reset()
    assert rel_l2(outs[1].cpu().numpy(), outs[0].cpu().numpy()) < (1e-10 if prec == "f64" else 1e-6)


@pytest.mark.parametrize("N,C", [(64, 3), (128, 2), (256, 1)])
@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("scheme", ["reference", "exact"])
def test_reverse_pass(small_stream, N, C, prec, scheme):
    """Both schemes against the whole GPU, to the engine's gradient tolerances."""
    import torch
    from cmblensing_b200 import _native as nat
    B, n = 2, 3
    plan, f, phi = _problem(torch, N, C, B, prec)
    lib, planes, cot = plan._lib, plan.phi_planes(phi), f.flip(-1).contiguous()
    io = nat.LF_F64 if prec == "f64" else nat.LF_F32
    nbytes = lib.lf_vjp_ckpt_workspace_bytes(plan.handle, B, n) if scheme == "exact" \
        else lib.lf_vjp_workspace_bytes(plan.handle, B)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    got = []
    torch.cuda.synchronize()
    for stream in (torch.cuda.current_stream(), small_stream):
        df, other = torch.empty_like(f), torch.empty_like(f)
        dphi = torch.empty((B, N, N), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        st = ctypes.c_void_p(stream.cuda_stream)
        if scheme == "exact":
            nat.check(lib.lf_lense_flow_vjp_ckpt(plan.handle, ptr(f), ptr(cot), io, ptr(planes), B, n, 1, ptr(other),
                                                 ptr(df), ptr(dphi), nat.LF_PHI_MAP, ptr(ws), nbytes, st))
        else:
            nat.check(lib.lf_lense_flow_vjp(plan.handle, ptr(f), ptr(cot), io, ptr(planes), B, n, 1, ptr(df), ptr(other),
                                            ptr(dphi), nat.LF_PHI_MAP, ptr(ws), nbytes, st))
        stream.synchronize()
        got.append([x.cpu().numpy() for x in (df, other, dphi)])
    for a, b in zip(*got):
        assert rel_l2(b, a) < (1e-9 if prec == "f64" else 2e-5)


def test_captured_lens(small_stream):
    """A graph captured on such a stream holds the stage launches."""
    import torch
    from cmblensing_b200 import engine
    B, n = 2, 2
    plan, f, phi = _problem(torch, 256, 2, B, "f32")
    planes = plan.phi_planes(phi)
    ws = torch.empty(plan.workspace_bytes(B, False, n), dtype=torch.uint8, device="cuda")
    want, out = torch.empty_like(f), torch.empty_like(f)
    torch.cuda.synchronize()
    with torch.cuda.stream(small_stream):
        plan.lense_flow(f, planes, n=n, out=want, workspace=ws)
    small_stream.synchronize()
    graph = engine.capture_graph(lambda: plan.lense_flow(f, planes, n=n, out=out, workspace=ws), stream=small_stream)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)

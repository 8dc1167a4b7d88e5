"""A wait that runs out ends a cluster's work: the blocks of the kernels for N <= 256 stop at the first one.

As in test_timeouts_gpu the hook lf_set_wait_polls(0) makes every first wait run out at once while the data are still
legitimately on their way; the drain wait keeps its limit, so nothing faults and nothing hangs."""
import time

import pytest

from oracle import lenseflow_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,B", [(64, 3), (128, 50), (256, 3)])
@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("kind", ["lens", "adjoint", "reverse", "exact reverse"])
def test_blocks_stop_at_the_first_timeout(N, B, prec, kind):
    """Nothing is written after the timeout, the call ends at once, and after the reset it computes as before."""
    import ctypes
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cmblensing_b200 import _native as nat
    from cmblensing_b200 import engine
    from cmblensing_b200.simulate import lens_batch
    lib = nat.load()
    C, n = 2, 3
    f, phis = lens_batch(N, 3.0, 2, C, seed0=190)
    reps = [i % 2 for i in range(B)]
    plan = engine.get_plan(N, C, R.pix_width_of(3.0), prec)
    ft = torch.as_tensor(f, device="cuda", dtype=plan.dtype)[reps].contiguous()
    planes = plan.phi_planes(torch.as_tensor(phis, device="cuda")[reps].contiguous())
    dphi = torch.empty((B, N, N), dtype=torch.float64, device="cuda")
    io = nat.LF_F64 if prec == "f64" else nat.LF_F32
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    nbytes = {"lens": plan.workspace_bytes(B, False, n), "adjoint": plan.workspace_bytes(B, True, n),
              "reverse": lib.lf_vjp_workspace_bytes(plan.handle, B),
              "exact reverse": lib.lf_vjp_ckpt_workspace_bytes(plan.handle, B, n)}[kind]
    ws = torch.zeros(nbytes, dtype=torch.uint8, device="cuda")

    def run(out):
        if kind in ("lens", "adjoint"):
            nat.check(lib.lf_lense_flow(plan.handle, ptr(ft), io, ptr(out), io, ptr(planes), B, n, 1,
                                        int(kind == "adjoint"), ptr(ws), nbytes, st))
        elif kind == "reverse":
            nat.check(lib.lf_lense_flow_vjp(plan.handle, ptr(ft), ptr(ft), io, ptr(planes), B, n, 1, ptr(out), None,
                                            ptr(dphi), nat.LF_PHI_MAP, ptr(ws), nbytes, st))
        else:
            nat.check(lib.lf_lense_flow_vjp_ckpt(plan.handle, ptr(ft), ptr(ft), io, ptr(planes), B, n, 1, None, ptr(out),
                                                 ptr(dphi), nat.LF_PHI_MAP, ptr(ws), nbytes, st))
        torch.cuda.synchronize()

    good, got = torch.empty_like(ft), torch.full_like(ft, 7.0)
    run(good)
    assert engine.wait_timeouts(reset=True) == 0
    try:
        nat.check(lib.lf_set_wait_polls(0), "lf_set_wait_polls")
        t0 = time.perf_counter()
        run(got)
        assert time.perf_counter() - t0 < 0.5
        assert engine.wait_timeouts() == 1
    finally:
        nat.check(lib.lf_set_wait_polls(-1), "lf_set_wait_polls")
        engine.wait_timeouts(reset=True)
    assert bool((got == 7.0).all())
    run(got)
    assert engine.wait_timeouts() == 0 and torch.equal(got, good)

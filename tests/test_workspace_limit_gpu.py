"""A lens whose p planes do not fit in memory takes the small workspace."""
import pytest

from oracle import lenseflow_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("captured", [False, True])
def test_no_room_for_p_planes(prec, captured):
    """The allocator may give out the small workspace and a quarter of the large one: the call runs, with the bits of
    the path that forms p in every stage; also inside a graph capture."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cmblensing_b200 import engine
    from cmblensing_b200.simulate import lens_batch
    N, C, B, n = 256, 1, 16, 10
    f, phis = lens_batch(N, 3.0, 2, C, seed0=210)
    reps = [i % 2 for i in range(B)]
    plan = engine.get_plan(N, C, R.pix_width_of(3.0), prec)
    ft = torch.as_tensor(f, device="cuda", dtype=plan.dtype)[reps].contiguous()
    planes = plan.phi_planes(torch.as_tensor(phis, device="cuda")[reps].contiguous())
    small, large = plan.workspace_bytes(B, False), plan.workspace_bytes(B, False, n)
    assert large > 4 * small
    out = torch.empty_like(ft)
    want = plan.lense_flow(ft, planes, n=n, workspace=torch.empty(small, dtype=torch.uint8, device="cuda"))
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + small + large // 4) / total)
    try:
        with pytest.raises(torch.OutOfMemoryError):
            torch.empty(large, dtype=torch.uint8, device="cuda")
        if captured:
            graph = engine.capture_graph(lambda: plan.lense_flow(ft, planes, n=n, out=out))
            graph.replay()
        else:
            plan.lense_flow(ft, planes, n=n, out=out)
        torch.cuda.synchronize()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.equal(out, want)

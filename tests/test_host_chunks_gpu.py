"""How a HostPipeline call is split: an explicit number is taken, the default depends on the bytes."""
import pytest

from oracle import lenseflow_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunks", [None, 1, 7, 8, 9])
def test_chunks(chunks):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cmblensing_b200 import engine
    plan = engine.get_plan(64, 1, R.pix_width_of(3.0))
    pipe = engine.HostPipeline(plan, 63, chunks=chunks)
    want = engine.default_chunks(pipe.h2d_bytes()) if chunks is None else chunks
    assert pipe.sizes == engine.chunk_schedule(63, want)
    assert len(pipe.sizes) == {None: want, 1: 1, 7: 7, 8: 8, 9: 9}[chunks]
    assert chunks is not None or want < 8

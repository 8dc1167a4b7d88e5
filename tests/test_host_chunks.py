"""The default split of a HostPipeline call, on the CPU."""
from cmblensing_b200.engine import chunk_schedule, default_chunks, default_schedule


def test_default_schedule_is_not_five_or_seven_chunks():
    """Where the batch divides so: six or eight; the other counts are default_chunks' own."""
    for batch in list(range(1, 130)) + [256, 1000]:
        for mb in (0, 1, 5, 12, 25, 38, 45, 50, 60, 75, 90, 100, 105, 115, 150, 400):
            sizes = default_schedule(batch, mb * 1e6)
            assert sum(sizes) == batch and min(sizes) > 0
            plain = chunk_schedule(batch, default_chunks(mb * 1e6))
            if len(plain) in (5, 7):
                assert sizes == chunk_schedule(batch, len(plain) + 1)
            else:
                assert sizes == plain
    assert len(default_schedule(128, 50e6)) == 6 and len(default_schedule(100, 105e6)) == 8
    assert len(default_schedule(12, 50e6)) == 4

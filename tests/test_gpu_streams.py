"""A context may be given another stream between any two calls: what the earlier ones enqueued is done."""
import pytest

pytestmark = pytest.mark.gpu


def test_set_stream_between_upload_and_fill(built_extension):
    import torch
    import morello_b200 as m
    plain = m.SynthesisDatabase(device=0)
    want = {}
    for size in (2, 4):
        plain.precompute(size)
        want[size] = plain.checksum()
    plain.close()
    db = m.SynthesisDatabase(device=0)
    streams = [torch.cuda.Stream() for _ in range(4)]
    for k, size in enumerate((4, 2, 4, 2)):   # the kept buffers hold the stages of the other size
        db.plan_precompute(size)
        db.upload()
        db.set_stream(streams[k].cuda_stream)
        db.fill()
        assert db.checksum() == want[size]
    db.close()

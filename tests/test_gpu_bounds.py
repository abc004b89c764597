"""Tables solved with pruned records and merged stage launches satisfy the defining recurrence: the
verifier evaluates every record at sampled limits, with no bound and no order."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,dtypes,shape", [
    ("MOVE", ("F32",), [16, 8]),          # more same-stage records than a batch holds
    ("MOVE", ("U32", "F32"), [1, 4, 16]),
    ("MATMUL", ("F32",), [1, 4, 8, 4]),   # grids of several work items, records that never fit
    ("MATMUL", ("U32", "F32"), [2, 1, 8, 2]),
    ("MATMUL_ACCUM", ("U32",), [1, 1, 32, 2]),
    ("MATMUL", ("U32",), [1, 1, 2, 1]),   # only small stages: one launch, no bounds
])
def test_tables_satisfy_the_recurrence(kind, dtypes, shape):
    import morello_b200 as m
    db = m.SynthesisDatabase(device=0)
    got = db.top_down_many([m.simple_spec(getattr(m, "KIND_" + kind), getattr(m, "DTYPE_" + d), shape, m.GL) for d in dtypes])
    assert all(d.found == 1 for d in got)
    checked, bad = db.verify(20_000_000, seed=3)
    assert checked == 20_000_000 and bad == 0
    db.close()

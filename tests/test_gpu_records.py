"""Calls that read the device's candidate records find all of them there: records planned on the host go
up in the background, and a table that was loaded from a file can be complete before they are."""
import pytest

pytestmark = pytest.mark.gpu


def test_get_impl_of_a_loaded_table_waits_for_the_records(built_extension, tmp_path):
    import morello_b200 as m
    path = str(tmp_path / "p4.mrldb")
    goals = [m.simple_spec(kind, m.DTYPE_F32, [1, 4, 4, 4][4 - rank:], m.GL)
             for kind, rank in ((m.KIND_MATMUL, 4), (m.KIND_MATMUL_ACCUM, 4), (m.KIND_MOVE, 3))]
    db = m.SynthesisDatabase(device=0)
    db.precompute(4)
    want = [db.get_impl(g) for g in goals]
    db.save(path)
    # the records of another job are what an early read would find in the kept buffer
    db.set_plan_flags(on_host=True, small_start=True)
    db.plan_precompute(2)
    db.upload()
    db.plan_precompute(4)
    db.load(path)          # uploads the plan, 280 MB of records in 64 KB pieces, and then the table
    assert [db.get_impl(g) for g in goals] == want
    checked, bad = db.verify(1_000_000)
    assert checked == 1_000_000 and bad == 0
    db.close()

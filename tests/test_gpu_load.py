"""Loading a saved table into a context with a plan. Calls that read the device's candidate records find
all of them there: records planned on the host go up in the background, and a loaded table can be complete
before they are. A file that is not sound replaces nothing."""
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


@pytest.mark.parametrize("on_host", [False, True])
@pytest.mark.parametrize("byte,value", [(1, 6), (3, 200)])   # of the first Spec's blob: another dtype; a rank there is not
def test_a_file_with_other_specs_replaces_nothing(built_extension, tmp_path, on_host, byte, value):
    import struct
    import morello_b200 as m
    db = m.SynthesisDatabase(device=0)
    db.set_plan_flags(on_host=on_host)
    db.precompute(1, dtypes=(m.DTYPE_U32,))
    path = str(tmp_path / "p1.mrldb")
    db.save(path)
    specs = [db.spec_blob(i) for i in range(db.num_specs())]
    want = db.get_many(specs, [m.MAX_MEM] * len(specs))
    data = bytearray(open(path, "rb").read())
    n_specs, = struct.unpack_from("<Q", data, 40)
    assert n_specs == len(specs)
    data[80 + 4 * n_specs + byte] = value
    open(path, "wb").write(data)
    db.plan_precompute(2, dtypes=(m.DTYPE_U32,))     # any other job: the file is not its own
    db.upload()
    db.fill()
    two = (db.checksum(), db.families())
    with pytest.raises(RuntimeError) as e:
        db.load(path)
    assert e.value.status == -8
    assert (db.checksum(), db.families()) == two
    checked, bad = db.verify(100_000)
    assert checked == 100_000 and bad == 0
    assert db.get_many(specs, [m.MAX_MEM] * len(specs)) == want   # Specs of size 1 are among those of size 2
    db.close()

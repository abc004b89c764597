"""The accessors of a plan made on the device: any number of threads may call them, and they answer from
the plan itself."""
import threading
import time

import pytest

pytestmark = pytest.mark.gpu


def test_first_accesses_from_several_threads(built_extension):
    import morello_b200 as m
    host = m.SynthesisDatabase(device=-1)
    host.plan_precompute(2)
    n = host.num_specs()
    want = [host.spec_blob(i) for i in range(n)]
    fams, stages = host.families(), host.stages()
    for _ in range(5):
        db = m.SynthesisDatabase(device=0)
        db.plan_precompute(2)
        wrong, gate = [], threading.Barrier(8)

        def work(t):
            gate.wait()
            if t % 4 == 3 and (db.families() != fams or db.stages() != stages):
                wrong.append("families")
            if [db.spec_blob(i) for i in range(n - 1, -1, -1)] != want[::-1]:
                wrong.append(t)

        threads = [threading.Thread(target=work, args=(t,)) for t in range(8)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        db.close()
        assert not wrong
    host.close()


def test_stages_and_families_need_no_host_plan(built_extension):
    import morello_b200 as m
    db, host = m.SynthesisDatabase(device=0), m.SynthesisDatabase(device=-1)
    goals = [m.simple_spec(m.KIND_MATMUL, m.DTYPE_F32, [2, 1, 8, 2], m.GL), m.simple_spec(m.KIND_MOVE, m.DTYPE_U32, [4, 8], m.GL)]
    for plan in (lambda d: d.plan_precompute(4), lambda d: d.plan_goals(goals)):
        plan(db)
        plan(host)
        t = time.perf_counter()
        got = db.stages(), db.families()
        t = time.perf_counter() - t
        assert got == (host.stages(), host.families())
        assert db.spec_owners() == host.spec_owners()
        if db.num_specs() > 100_000:   # a host plan of these takes as long as the one beside it
            assert t < host.stats()["plan_seconds"] / 2
    db.close()
    host.close()

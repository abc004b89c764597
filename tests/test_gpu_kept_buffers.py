"""A context's device buffers stay from plan to plan: what they hold or how large they are from before has
no bearing on the next plan's tables, on what the context keeps, or on what it can do."""
import pytest

pytestmark = pytest.mark.gpu


def _jobs(m):
    u, f = m.DTYPE_U32, m.DTYPE_F32
    goal = lambda *a: lambda d: d.plan_goals([m.simple_spec(*a, m.GL)])
    return {
        "precompute 4": lambda d: d.plan_precompute(4),                       # more Specs than merged launches take
        "1x1x1": goal(m.KIND_MATMUL, u, [1, 1, 1, 1]),
        "relayout": goal(m.KIND_MOVE, f, [16, 16]),
        "size-8 Moves": lambda d: d.plan_precompute(8, m.THROUGH_MOVE, (f,)),
        "8x8x8": goal(m.KIND_MATMUL, f, [1, 8, 8, 8]),
        "precompute 2": lambda d: d.plan_precompute(2),
    }


def _used(torch, base):
    torch.cuda.synchronize()
    return base - torch.cuda.mem_get_info()[0]


def test_jobs_of_many_sizes_in_one_context(built_extension):
    import torch
    import morello_b200 as m
    jobs = _jobs(m)
    want, fresh = {}, {}
    m.SynthesisDatabase(device=0).close()
    for name, plan in jobs.items():
        base = torch.cuda.mem_get_info()[0]
        db = m.SynthesisDatabase(device=0)
        plan(db)
        db.upload()
        db.fill()
        want[name] = (db.stats()["n_candidates"], db.checksum())
        fresh[name] = _used(torch, base)
        db.close()
    base = torch.cuda.mem_get_info()[0]
    db = m.SynthesisDatabase(device=0)
    for name, on_host in (("precompute 4", False), ("1x1x1", False), ("precompute 4", False), ("precompute 2", True), ("size-8 Moves", False),
                          ("precompute 2", False), ("8x8x8", False), ("1x1x1", True), ("precompute 4", True), ("relayout", False)):
        db.set_plan_flags(on_host=on_host)
        jobs[name](db)
        db.upload()
        db.fill()
        assert (db.stats()["n_candidates"], db.checksum()) == want[name], (name, on_host)
    # the relayout's 0.4 GB after the 2.4 of precompute 4
    assert _used(torch, base) < fresh["relayout"] + (1 << 30)
    db.close()


def test_what_a_context_keeps_is_not_in_its_own_way(built_extension):
    import torch
    import morello_b200 as m
    jobs = _jobs(m)
    solo = m.SynthesisDatabase(device=0)
    jobs["8x8x8"](solo)
    solo.upload()
    solo.fill()
    want = solo.checksum()
    solo.close()
    db = m.SynthesisDatabase(device=0)
    jobs["size-8 Moves"](db)      # 2.2 GB of working rows, 0.3 of table, 0.3 of records
    db.upload()
    db.fill()
    torch.cuda.synchronize()
    rest = torch.empty(torch.cuda.mem_get_info()[0] - (24 << 20), dtype=torch.uint8, device="cuda")
    try:
        jobs["8x8x8"](db)         # more records, fewer working rows
        db.upload()
        db.fill()
        assert db.checksum() == want
    finally:
        del rest
        torch.cuda.empty_cache()
        db.close()


@pytest.mark.parametrize("kind,dtypes,shape", [
    ("MATMUL", ("U32",), [1, 2, 2, 2]),           # one launch of all stages, by a block
    ("MATMUL", ("U32", "F32"), [1, 2, 8, 4]),     # launches of several stages, by teams of all sizes
    ("MOVE", ("F32",), [16, 16]),
])
def test_fills_that_enlarge_their_buffers(built_extension, kind, dtypes, shape):
    import morello_b200 as m
    goals = [m.simple_spec(getattr(m, "KIND_" + kind), getattr(m, "DTYPE_" + d), shape, m.GL) for d in dtypes]
    solo = m.SynthesisDatabase(device=0)
    want = solo.top_down_many(goals)
    assert solo.stats()["n_buffer_growths"] == 0
    for on_host in (False, True):
        db = m.SynthesisDatabase(device=0)
        db.set_plan_flags(on_host=on_host, small_start=True)
        assert db.top_down_many(goals) == want
        assert db.stats()["n_buffer_growths"] > 0
        assert db.checksum() == solo.checksum()
        db.fill()                                  # the enlarged buffers stay
        assert db.stats()["n_buffer_growths"] == 0 and db.checksum() == solo.checksum()
        db.close()
    solo.close()

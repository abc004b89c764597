"""The stage-by-stage fill of two ranks, one after the other on one GPU (no kernel waits for another
rank): solving, the sum of the masks, placing and the sum of the rows give the unsharded table."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [2, 4])
def test_two_ranks_in_turn_equal_one_fill(size):
    import torch
    import morello_b200 as m
    from morello_b200 import sharded
    solo = m.SynthesisDatabase(device=0)
    solo.precompute(size)
    ranks = []
    for r in range(2):
        db = m.SynthesisDatabase(device=0)
        db.set_shard(r, 2)
        db.plan_precompute(size)
        db.upload()
        db.fill_begin()
        ranks.append(db)

    def words(ptr, nbytes):
        return torch.as_tensor(sharded._DeviceBytes(ptr, nbytes), device="cuda").view(torch.int32)

    def exchange(parts):
        total = parts[0] + parts[1]
        for p in parts:
            p.copy_(total)
        torch.cuda.synchronize()

    for s in range(ranks[0].num_stages()):
        got = [db.fill_stage_solve(s) for db in ranks]
        exchange([words(*g) for g in got])
        rows = [db.fill_stage_place(s) for db in ranks]
        assert rows[0][1] == rows[1][1]
        exchange([words(*g) for g in rows])
    for db in ranks:
        db.fill_end()
        assert db.checksum() == solo.checksum() and db.stats()["n_rows"] == solo.stats()["n_rows"]
        db.close()
    solo.close()

"""Plans made on the device equal the host planner's, record for record and Spec for Spec."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _goals(m):
    # ragged shapes, a batch, ranks 1 to 4, both dtypes with different goal sets, every kind; and
    # operands in fast memories
    return {
        "mixed": [m.simple_spec(m.KIND_MATMUL, m.DTYPE_F32, [2, 1, 8, 2], m.GL), m.simple_spec(m.KIND_MOVE, m.DTYPE_U32, [2, 2, 2, 2], m.GL),
                  m.simple_spec(m.KIND_FILL_ZERO, m.DTYPE_U32, [16], m.L1), m.simple_spec(m.KIND_MATMUL_ACCUM, m.DTYPE_U32, [1, 4, 1, 2], m.RF)],
        "one": [m.simple_spec(m.KIND_MOVE, m.DTYPE_F32, [1], m.RF)],
        "relayouts": [m.simple_spec(m.KIND_MOVE, m.DTYPE_F32, [32, 8], m.GL)],
        "long": [m.simple_spec(m.KIND_MOVE, m.DTYPE_U32, [512], m.GL)],   # a dimension of two key bytes
    }


@pytest.mark.parametrize("job", ["mixed", "one", "relayouts", "long", (1, 0), (2, 2), (4, 1), (4, 2), (8, 1)])
def test_device_plan_equals_host_plan(job):
    import torch
    import morello_b200 as m
    db, host = m.SynthesisDatabase(device=0), m.SynthesisDatabase(device=-1)
    for d in (db, host):
        if isinstance(job, str):
            d.plan_goals(_goals(m)[job])
        else:
            d.plan_precompute(job[0], job[1])
    a, b = db.stats(), host.stats()
    assert a["plan_layout_seconds"] == 0 and b["plan_layout_seconds"] > 0   # only the host planner lays ids out
    for k in ("n_specs", "n_goal_specs", "n_candidates", "n_stages"):
        assert a[k] == b[k], k
    db.upload()
    ptr, nbytes = db.device_cands()

    class Records:
        __cuda_array_interface__ = {"shape": (nbytes,), "typestr": "|u1", "data": (ptr, False), "strides": None, "version": 3}

    got = torch.as_tensor(Records(), device=torch.device("cuda", 0)).cpu().numpy()
    want = np.frombuffer(ctypes.string_at(*host.plan_share()[3]), dtype=np.uint8)
    assert got.size == want.size and (got == want).all()
    step = max(1, db.num_specs() // 5000)
    for i in range(0, db.num_specs(), step):
        assert db.spec_blob(i) == host.spec_blob(i)
    assert db.stages() == host.stages()
    db.close()
    host.close()

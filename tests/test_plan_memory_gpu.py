"""Device memory of reusable plans."""
import numpy as np
import pytest

from qspace_gb300.grouped import DeviceBatch, Packed


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["fp64", "split"])
def test_a_second_plan_maps_no_new_memory(prec):
    """A plan's lists and digits come from the context's pool: a plan created
    after another of its size was destroyed reuses that memory, which neither
    mapping nor unmapping then delays."""
    rng = np.random.default_rng(0)
    shapes = [(700, 600, 500), (300, 2, 3), (900, 1000, 40), (64, 64, 64)]
    pk = Packed([rng.standard_normal((m, k)) for m, n, k in shapes], [rng.standard_normal((k, n)) for m, n, k in shapes],
                np.ones(len(shapes)))
    db = DeviceBatch(pk)
    ref = None
    free = []
    for _ in range(4):
        plan = db.plan(prec, graph=False)
        db.ctx.sync()
        free.append(db.torch.cuda.mem_get_info()[0])
        db.dC.fill_(float("nan"))
        db.torch.cuda.synchronize()
        db.run_plan(plan)
        got = db.result()
        ref = ref or [c.copy() for c in got]
        assert all(np.array_equal(c, r) for c, r in zip(got, ref))
        plan.close()
        db.ctx.sync()
        free.append(db.torch.cuda.mem_get_info()[0])
    assert len(set(free[2:])) == 1, free

"""Runs in one stream begin while their predecessor drains: each must still see
its predecessor's memory (keys written, answers read, scratch shared) and no
run may overtake another, in a stream and in a captured graph."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 700, 40_000, 2_000_003])
@pytest.mark.parametrize("graph", [False, True])
def test_chained_runs(n, graph):
    from apsep_gb300 import Plan
    rng = np.random.default_rng(n)
    a = rng.integers(0, 1 << 30, n).astype(np.int32)
    x0 = torch.from_numpy(a).cuda()
    steps = 6
    bufs = [torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(steps)]
    keys = [torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(steps)]
    with Plan(n, torch.int32) as plan:
        def chain():  # each run's keys come from the answers before it, through the run's own plan
            cur = x0
            for s in range(steps):
                plan.run(cur, out=bufs[s])
                torch.bitwise_xor(bufs[s], x0, out=keys[s])
                cur = keys[s]
        chain()
        plan.check()
        if graph:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                chain()
            for b in bufs:
                b.fill_(-7)
            for _ in range(3):
                g.replay()
            plan.check()
        got = [b.cpu().numpy() for b in bufs]
    cur = a
    for s in range(steps):
        want = oracle.apse(cur, False)
        assert np.array_equal(got[s], want), s
        cur = want ^ a


def test_back_to_back_runs_on_one_plan():
    from apsep_gb300 import Plan
    rng = np.random.default_rng(3)
    arrays = [rng.integers(0, 50 if k % 2 else 1 << 30, 60_000 + 977 * k).astype(np.int32) for k in range(40)]
    xs = [torch.from_numpy(a).cuda() for a in arrays]
    with Plan(120_000, torch.int32) as plan:
        outs = [plan.run(x) for x in xs]
        plan.check()
    for a, o in zip(arrays, outs):
        assert np.array_equal(o.cpu().numpy(), oracle.apse(a, False))

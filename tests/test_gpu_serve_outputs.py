"""The pool server writes a request's answers where its `out` points when its batch
is launched: on_done may have given a later request another buffer by then."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("device", ["cuda", "cpu"])
def test_outputs_set_while_serving(device):
    from apsep_gb300.serve import PoolServer, Request
    n, count = 4000, 24
    rng = np.random.default_rng(5)
    keys = [rng.integers(0, 1 << 30, n).astype(np.int32) for _ in range(count)]
    first = torch.full((count, n), -7, dtype=torch.int32, device="cuda")
    reqs = [Request(rid=i, keys=torch.from_numpy(k).cuda(), out=first[i]) for i, k in enumerate(keys)]
    last = torch.full((n,), -7, dtype=torch.int32, device=device)
    if device == "cpu":
        last = last.pin_memory()

    def on_done(r, answers):
        if r.rid == 0:  # a batch holds one request: the last one is far from its launch
            reqs[-1].out = last

    server = PoolServer(budget_bytes=64 << 20, kinds=((torch.int32, False),), max_batch_keys=n, ring_keys=4 * n)
    try:
        server.serve(reqs, realtime=False, on_done=on_done)
    finally:
        server.close()
    torch.cuda.synchronize()
    got = first.cpu().numpy()
    for i in range(count - 1):
        assert np.array_equal(got[i], oracle.apse(keys[i])), i
    assert np.array_equal(last.cpu().numpy(), oracle.apse(keys[-1]))
    assert (got[-1] == -7).all()

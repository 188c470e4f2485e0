"""Consumers over 8-byte keys in the arrays whose flips and reversals the
engine does itself, from the shortest such array on, against the CPU oracles
(of the keys' ranks: the same order in int32)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import consumers as oc  # noqa: E402
from test_gpu_structured import keys, ranked  # noqa: E402

pytestmark = pytest.mark.gpu


def _keys(shape, n, dtype):
    rng = np.random.default_rng(n)
    if shape == "uniform":
        a = rng.integers(-(1 << 62), 1 << 62, n)
    elif shape == "few":  # both signs of zero among the float keys
        a = rng.integers(-2, 3, n)
    elif shape == "walk":
        a = keys("walk", n, n) - 12345
    else:
        a = keys(shape, n, n) - n // 2
    x = a.astype(dtype)
    if dtype == "float64":
        x[::3] *= -1.0 if shape == "few" else 1.0
    return x


@pytest.mark.parametrize("dtype", ["int64", "float64"])
@pytest.mark.parametrize("shape", ["uniform", "few", "walk", "down_few", "up_few"])
def test_wide_consumers(shape, dtype):
    from apsep_gb300 import Plan, consumers
    edge = 256 * 8 * torch.cuda.get_device_properties(0).multi_processor_count
    with Plan(edge + 800_000, getattr(torch, dtype)) as plan:
        for n in (edge, edge + 1, edge + 32, edge + 33, edge + 480, edge + 512, edge + 543, edge + 700_015):
            a = _keys(shape, n, dtype)
            x, r = torch.from_numpy(a).cuda(), ranked(a)
            for le in (False, True):
                got = consumers.prev_greater(x, inclusive=le, plan=plan).cpu().numpy()
                assert np.array_equal(got, oc.prev_greater(r, le)), (n, le)
                got = consumers.next_smaller(x, inclusive=le, plan=plan).cpu().numpy()
                assert np.array_equal(got, oc.next_smaller(r, le)), (n, le)
            assert np.array_equal(consumers.stock_span(x, plan=plan).cpu().numpy(), oc.stock_span(r)), n
            assert np.array_equal(consumers.cartesian_parents(x, plan=plan).cpu().numpy(), oc.cartesian_parents(r)), n
        plan.check()

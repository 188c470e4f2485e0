"""Consumers that look to the right, at lengths that are not whole rows of 32
keys: the last n % 32 keys answer, and are answered, apart from the engine's
reversed run.  Bit-exact against the CPU oracles."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import consumers as oc  # noqa: E402

pytestmark = pytest.mark.gpu

SIZES = [31, 32, 33, 63, 65, 511, 543, 4097, 70_001, 1_000_031]


def keys(shape: str, n: int) -> np.ndarray:
    rng = np.random.default_rng(n)
    if shape == "uniform":
        return rng.integers(0, 1 << 20, n)
    if shape == "few_values":
        return rng.integers(0, 4, n)
    if shape == "falling":  # every answer is the next key, across the boundary too
        return np.arange(n, 0, -1)
    a = np.arange(n) + 64  # rising: no answers before the last keys
    a[-(n % 32 or 1):] = rng.integers(0, n + 64, n % 32 or 1)  # the tail answers many at once
    return a


@pytest.mark.parametrize("shape", ["uniform", "few_values", "falling", "rising_tail"])
@pytest.mark.parametrize("dtype", ["int32", "float32"])
def test_tails(shape, dtype):
    from apsep_gb300 import Plan, consumers
    with Plan(max(SIZES), getattr(torch, dtype)) as plan:
        for n in SIZES:
            a = keys(shape, n).astype(dtype)
            x = torch.from_numpy(a).cuda()
            for le in (False, True):
                got = consumers.next_smaller(x, inclusive=le, plan=plan).cpu().numpy()
                assert np.array_equal(got, oc.next_smaller(a, le)), (shape, dtype, n, le)
            got = consumers.cartesian_parents(x, plan=plan).cpu().numpy()
            assert np.array_equal(got, oc.cartesian_parents(a)), (shape, dtype, n)
            if dtype == "int32":
                assert consumers.largest_rectangle(x, plan=plan) == oc.largest_rectangle(a), (shape, n)
        plan.check()

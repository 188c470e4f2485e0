"""Keys of the pads' values -- the largest of their type, and for flipped runs the
smallest; infinities -- through every form of the engine that reads its keys
through a map or from the end: the pads before a tile's first lane, the window and
the prefix minimum all compare equal to them under <=.  Against the CPU oracles (of
the keys' ranks)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402
from oracle import consumers as oc  # noqa: E402
from test_gpu_structured import ranked  # noqa: E402

pytestmark = pytest.mark.gpu


def _keys(shape, n, dtype):
    rng = np.random.default_rng(n)
    lo, hi = (-np.inf, np.inf) if dtype.startswith("float") else (np.iinfo(dtype).min, np.iinfo(dtype).max)
    some = np.array([hi, lo, 7, -7, 0], dtype=dtype)
    if shape == "hi":
        return np.full(n, hi, dtype=dtype)
    if shape == "lo":
        return np.full(n, lo, dtype=dtype)
    if shape == "mix":
        return rng.choice(some, n, p=[.6, .05, .15, .15, .05])
    if shape == "runs":  # runs of one value, whole tiles of them
        ends = np.cumsum(rng.integers(1, 4097, n // 1024 + 2))
        return rng.choice(some, ends.size + 1, p=[.45, .25, .1, .1, .1])[np.searchsorted(ends, np.arange(n), side="right")]
    # falling keys from the largest value down to the smallest, in runs, ties at both ends
    i = np.arange(n) % 3000
    a = ((1500 - i) * 1000).astype(dtype)
    a[i < 40] = hi
    a[i > 2950] = lo
    return a


def _sizes(dtype):
    if dtype in ("int64", "float64"):  # the long tiles, from their first length on
        edge = 256 * 8 * torch.cuda.get_device_properties(0).multi_processor_count
        return edge, edge + 32, edge + 543, edge + 300_031
    return 32, 480, 543, 4096, 70_001, 1_000_032, 1_000_063


@pytest.mark.parametrize("dtype", ["int32", "float32", "int64", "float64"])
@pytest.mark.parametrize("shape", ["hi", "lo", "mix", "runs", "falling"])
def test_pad_keys(shape, dtype):
    from apsep_gb300 import Plan, consumers
    sizes = _sizes(dtype)
    with Plan(max(sizes), getattr(torch, dtype)) as plan:
        for n in sizes:
            a = _keys(shape, n, dtype)
            x, r = torch.from_numpy(a).cuda(), ranked(a)
            for le in (False, True):
                got = plan.run(x, inclusive=le).cpu().numpy()
                assert np.array_equal(got, oracle.apse(r, le)), ("run", n, le)
                got = consumers.prev_greater(x, inclusive=le, plan=plan).cpu().numpy()
                assert np.array_equal(got, oc.prev_greater(r, le)), ("greater", n, le)
                got = consumers.next_smaller(x, inclusive=le, plan=plan).cpu().numpy()
                assert np.array_equal(got, oc.next_smaller(r, le)), ("next", n, le)
            assert np.array_equal(consumers.stock_span(x, plan=plan).cpu().numpy(), oc.stock_span(r)), n
            assert np.array_equal(consumers.cartesian_parents(x, plan=plan).cpu().numpy(), oc.cartesian_parents(r)), n
            if dtype == "int32":
                h = np.maximum(a, 0)
                assert consumers.largest_rectangle(torch.from_numpy(h).cuda(), plan=plan) == oc.largest_rectangle(h), n
        plan.check()


@pytest.mark.parametrize("dtype", ["int32", "float32", "int64", "float64"])
@pytest.mark.parametrize("shape", ["hi", "lo", "mix", "runs", "falling"])
def test_pad_keys_with_int64_positions(shape, dtype):
    from apsep_gb300 import Plan
    for n, piece in ((400_003, 131_072), (70_001, 70_001), (100_000, 1_024)):
        a = _keys(shape, n, dtype)
        x, r = torch.from_numpy(a).cuda(), ranked(a)
        for le in (False, True):
            with Plan(piece, getattr(torch, dtype), inclusive=le) as plan:
                got = plan.run64(x).cpu().numpy()
                plan.check()
            assert np.array_equal(got, oracle.apse(r, le)), (n, piece, le)

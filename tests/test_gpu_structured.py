"""Keys with structure, bit-exact against the oracle: random walks (many
prefix minima per range: deep stacks, long lists of deferred and capped
keys), sorted keys with a few out of place (one earlier key answers whole
tiles), ramps and noisy slopes (more cross-lane queries than one round)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402

pytestmark = pytest.mark.gpu


def keys(shape: str, n: int, seed: int) -> np.ndarray:
    rng = np.random.default_rng(seed)
    i = np.arange(n, dtype=np.int64)
    if shape == "walk":
        return np.cumsum(rng.integers(-1000, 1001, n))
    if shape == "walk_down":  # most keys are prefix minima
        return np.cumsum(rng.integers(-1000, 801, n))
    if shape == "ramps":
        return i % 257
    if shape == "falling_runs":  # descending runs of up to 4096 keys from random starts
        ends = np.cumsum(rng.integers(1, 4097, n // 1024 + 2))
        run = np.searchsorted(ends, i, side="right")
        return rng.integers(4096, 1 << 30, ends.size + 1)[run] - (i - np.concatenate([[0], ends])[run])
    if shape == "noisy_down":
        return 8 * (n - i) + rng.integers(0, 64, n)
    x = i.copy() if shape == "up_few" else n - 1 - i
    at = rng.integers(0, n, max(1, n // 5000))
    x[at] = rng.integers(0, n, at.size)
    return x


SHAPES = ("walk", "walk_down", "ramps", "falling_runs", "noisy_down", "down_few", "up_few")


def ranked(a: np.ndarray) -> np.ndarray:
    """The same order in int32 (the oracle's integer keys)."""
    return np.unique(a, return_inverse=True)[1].astype(np.int32)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dtype", ["int32", "float32", "int64", "float64"])
@pytest.mark.parametrize("le", [False, True])
def test_single_array(shape, dtype, le):
    from apsep_gb300 import Plan
    dt = getattr(torch, dtype)
    for n in (511, 2049, 70_001, 1_300_000, 3 << 20):
        a = keys(shape, n, n + 7)
        x = torch.from_numpy(a.astype(dtype)).cuda()
        want = oracle.apse(ranked(x.cpu().numpy()), le)
        with Plan(n, dt, inclusive=le) as plan:
            got = plan.run(x)
            plan.check()
        assert np.array_equal(got.cpu().numpy(), want), (shape, dtype, le, n)


@pytest.mark.parametrize("shape", SHAPES)
def test_every_configuration(shape):
    from apsep_gb300 import Plan, autotune
    n = 1_100_003
    a = keys(shape, n, 3).astype(np.int32)
    want = oracle.apse(a, False)
    x = torch.from_numpy(a).cuda()
    with Plan(n, torch.int32, tuning=None) as plan:
        for cfg in range(autotune.num_configs()):
            plan.set_config(cfg)
            got = plan.run(x)
            plan.check()
            assert np.array_equal(got.cpu().numpy(), want), (shape, cfg)


@pytest.mark.parametrize("dtype", ["int32", "float32", "int64"])
@pytest.mark.parametrize("le", [False, True])
def test_batch(dtype, le):
    from apsep_gb300 import Plan
    rng = np.random.default_rng(11)
    lens = [1, 3, 700, 33, 200_000, 0, 5, 41_003, 512, 300_000, 31, 90_001, 123_456, 64, 150_000, 77, 99_999]
    parts = [keys(SHAPES[k % len(SHAPES)], m, k) if m else np.zeros(0, np.int64) for k, m in enumerate(lens)]
    a = np.concatenate(parts) + rng.integers(0, 2)
    offs = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    x = torch.from_numpy(a.astype(dtype)).cuda()
    want = oracle.apse_segmented(ranked(x.cpu().numpy()), offs, le)
    with Plan(a.size, getattr(torch, dtype), inclusive=le) as plan:
        got = plan.run_segmented(x, torch.from_numpy(offs).cuda())
        plan.check()
    assert np.array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("shape", SHAPES)
def test_consumers_and_int64_positions(shape):
    from apsep_gb300 import Plan, consumers
    n = 800_000
    a = keys(shape, n, 5).astype(np.int32)
    x = torch.from_numpy(a).cuda()
    i = np.arange(n)
    prev_greater = oracle.apse(-a - 1, False)
    assert np.array_equal(consumers.prev_greater(x).cpu().numpy(), prev_greater)
    assert np.array_equal(consumers.stock_span(x).cpu().numpy(), i - prev_greater)
    r = oracle.apse(np.ascontiguousarray(a[::-1]), False)[::-1]
    assert np.array_equal(consumers.next_smaller(x).cpu().numpy(), np.where(r >= 0, n - 1 - r, -1))
    with Plan(300_000, torch.int32) as plan:
        got = plan.run64(x)
        plan.check()
    assert np.array_equal(got.cpu().numpy(), oracle.apse(a, False).astype(np.int64))

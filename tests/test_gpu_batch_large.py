"""Batches around the size at which configuration 0 gives them CTAs of their own (20
warps, shorter stack and lists): every form of that kernel -- key type, comparator,
keys off a 16-byte boundary -- and the last batch that still takes the other one,
over arrays that span many ranges and overflow the lists."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402
from test_gpu_structured import keys  # noqa: E402

pytestmark = pytest.mark.gpu

POISON = -1414812757
SHARES = [("walk", 0.30), ("walk_down", 0.25), ("down_few", 0.15), ("up_few", 0.05), ("falling_runs", 0.05),
          ("pads", 0.10), ("uniform", 1.0)]


def batch(n: int, dtype: str):
    """Arrays of the shapes above, a few tiny ones between them; n keys in all."""
    rng = np.random.default_rng(n)
    parts, left = [], n
    for shape, share in SHARES:
        for m in (min(left, int(share * n) if share < 1.0 else left), 0, 1, 33):
            m = min(m, left) if shape != "uniform" else left
            if shape == "uniform":
                a = rng.integers(0, 1 << 30, m).astype(dtype)
            elif shape == "pads":  # keys of the pad's value, the smallest value and a few others
                lo, hi = (-np.inf, np.inf) if dtype == "float32" else (np.iinfo(dtype).min, np.iinfo(dtype).max)
                a = rng.choice(np.array([hi, hi, hi, hi, 5, 3, lo], dtype=dtype), m, p=[.4, .3, .2, .07, .02, .0099, .0001])
            else:
                a = keys(shape, max(m, 2), m + 1)[:m].astype(dtype)
            parts.append(a)
            left -= m
            if left == 0:
                break
    offs = np.concatenate([[0], np.cumsum([p.size for p in parts])])
    assert offs[-1] == n
    return np.concatenate(parts), offs.astype(np.int64)


@pytest.mark.parametrize("dtype", ["int32", "float32"])
@pytest.mark.parametrize("tiles,past,shift", [(0, 0, 0), (0, 77, 1), (0, 0, 2), (0, 511, 3), (-1, 0, 0), (-1, -1, 1)])
def test_batches_around_the_change(dtype, tiles, past, shift):
    from apsep_gb300 import Plan
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = (6 * 20 * sms + tiles) * 512 + past  # six tiles a warp on 20 warps per SM
    a, offs = batch(n, dtype)
    xb = torch.zeros(n + 4, dtype=getattr(torch, dtype), device="cuda")
    xb[shift:shift + n] = torch.from_numpy(a).cuda()
    d_offs = torch.from_numpy(offs).cuda()
    for le in (False, True):
        ob = torch.full((n + 4,), POISON, dtype=torch.int32, device="cuda")
        with Plan(n, xb.dtype, inclusive=le) as plan:
            plan.set_config(0)
            plan.run_segmented(xb[shift:shift + n], d_offs, out=ob[shift:shift + n])
            plan.check()
        got = ob.cpu().numpy()
        want = oracle.apse_segmented(a, offs, le)
        bad = np.flatnonzero(got[shift:shift + n] != want)
        assert bad.size == 0, (le, bad.size, int(bad[0]), int(np.searchsorted(offs, bad[0], side="right") - 1))
        assert (got[:shift] == POISON).all() and (got[shift + n:] == POISON).all()

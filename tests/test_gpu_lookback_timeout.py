"""A range whose wait for its predecessors gives up takes nothing from them: their
words may be an older run's, with positions past this run's keys.  Keys equal to
the pad are the ones for which a minimum nobody published would qualify (<=)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("config", [0, 5])  # 48 ranges wait on one another, 96 on the count
@pytest.mark.parametrize("dtype,pad", [("int32", np.iinfo(np.int32).max), ("float32", np.inf)])
def test_keys_of_the_pads_value(dtype, pad, config):
    from apsep_gb300 import ApsepError, Plan, _lib
    n, skipped, tile = 4096 * 6, 2, 512 if config == 0 else 256
    long = torch.full((1 << 20,), pad, dtype=getattr(torch, dtype), device="cuda")
    with Plan(1 << 20, long.dtype, inclusive=True) as plan:
        plan.set_config(config)
        plan.run(long)  # leaves the words of a longer run
        plan.check()
        plan.debug_inject(range_index=skipped, spin_limit=2000)
        got = plan.run(long[:n])
        with pytest.raises(ApsepError) as ei:
            plan.check()
        assert ei.value.status == _lib.APSEP_ETIMEOUT
        want = np.arange(-1, n - 1)
        want[(skipped + 1) * tile::tile] = -1  # the first keys of the ranges that gave up
        assert np.array_equal(got.cpu().numpy(), want)
        got = plan.run(long[:n])  # the plan still works
        plan.check()
        assert np.array_equal(got.cpu().numpy(), oracle.apse(long[:n].cpu().numpy(), True))

"""8-byte keys: both lengths of their warp tiles, around the array length where
one gives way to the other and at the edges of the longer tile."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402
from test_gpu_structured import keys, ranked  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["int64", "float64"])
@pytest.mark.parametrize("shape", ["walk", "noisy_down", "up_few"])
@pytest.mark.parametrize("past", [0, 1, 15, 31, 511, 512, 513, 700_015])
def test_around_the_change(dtype, shape, past):
    from apsep_gb300 import Plan
    # one 8-warp CTA of 256-key tiles on every SM, the last length of the short tiles
    n = 256 * 8 * torch.cuda.get_device_properties(0).multi_processor_count + past
    a = keys(shape, n, n)
    if past % 2:
        a = np.random.default_rng(n).permutation(a)
    buf = torch.empty(n + 1, dtype=getattr(torch, dtype), device="cuda")
    for off in (0, 1):  # 1: 8 bytes past a 16-byte boundary, plain loads and stores
        buf[off:off + n] = torch.from_numpy(a.astype(dtype)).cuda()
        for le in (False, True):
            with Plan(n, buf.dtype, inclusive=le) as plan:
                got = plan.run(buf[off:off + n])
                plan.check()
            want = oracle.apse(ranked(buf[off:off + n].cpu().numpy()), le)
            assert np.array_equal(got.cpu().numpy(), want), (off, le)

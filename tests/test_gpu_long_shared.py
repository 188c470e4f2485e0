"""int64 positions: pieces whose keys share answers before the piece
(descending keys after a few low ones, pieces that fall while the array
rises, ties), bit-exact against the oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402
from test_gpu_structured import keys, ranked  # noqa: E402

pytestmark = pytest.mark.gpu


def _shape(kind, n, piece):
    i = np.arange(n, dtype=np.int64)
    if kind == "falling_pieces":  # every key of a piece is answered before it
        return i // piece * (piece // 2) - i % piece
    if kind == "steps":  # long runs of equal keys, going down
        return (n - i) // 1500
    if kind == "mountain":  # up, then down: an answer of its own for every key of the falling half
        return np.minimum(2 * i, 2 * (n - i) - 1) + i % 7
    return keys(kind, n, n)


@pytest.mark.parametrize("kind", ["down_few", "walk_down", "noisy_down", "falling_pieces", "steps", "mountain"])
@pytest.mark.parametrize("dtype", ["int32", "float32", "int64", "float64"])
@pytest.mark.parametrize("n,piece,off", [(70_001, 4096, 0), (70_001, 33_333, 1), (1_500_007, 511_999, 0),
                                         (3_000_000, 1 << 20, 1)])
def test_shared_answers(kind, dtype, n, piece, off):
    from apsep_gb300 import Plan
    buf = torch.empty(n + off, dtype=getattr(torch, dtype), device="cuda")
    x = buf[off:]
    x.copy_(torch.from_numpy(_shape(kind, n, piece).astype(dtype)))
    for le in (False, True):
        want = oracle.apse(ranked(x.cpu().numpy()), le).astype(np.int64)
        with Plan(piece, x.dtype, inclusive=le) as plan:
            got = plan.run64(x)
            plan.check()
        assert np.array_equal(got.cpu().numpy(), want), le

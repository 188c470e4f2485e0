"""Argument lists of the span copy's Python binding (no GPU): the C call reads as
many entries of each list as there are sources."""
import pytest

from apsep_gb300 import _lib


@pytest.mark.parametrize("srcs,dsts,nbytes", [([16, 32], [48], [0, 0]), ([16, 32], [48, 64], [0]), ([16], [48, 64], [0])])
def test_lists_of_different_lengths_are_refused(srcs, dsts, nbytes):
    with pytest.raises(ValueError):
        _lib.copy_spans(srcs, dsts, nbytes, 0)


def test_null_addresses_reach_the_library():
    if not _lib.os.path.isfile(_lib.LIB_PATH):
        pytest.skip("libapsep.so is not built")
    with pytest.raises(_lib.ApsepError) as ei:
        _lib.copy_spans([None], [16], [4], 0)  # bytes from nowhere
    assert ei.value.status == _lib.APSEP_EINVAL
    _lib.copy_spans([], [], [], 0)

"""Results around the lengths at which their download changes: one copy, pieces of 1 MiB, four pieces."""
import numpy as np
import pytest

from cuda_replace_b200.cuda_replace_wrapper import Session

pytestmark = pytest.mark.gpu

MiB = 1 << 20


@pytest.mark.parametrize("n", [1, 3 * MiB - 1, 3 * MiB, 4 * MiB - 1, 4 * MiB, 4 * MiB + 1, 5 * MiB - 7, 24 * MiB, 24 * MiB + 1, 33 * MiB + 5, 96 * MiB + 1])
def test_result_and_unified_into(cr_lib, n):
    base = np.random.default_rng(n).integers(0, 255, size=MiB + 13, dtype=np.uint8)
    src = np.resize(base, n).tobytes()
    with Session(cr_lib, src) as s:
        assert s.result() == src
        assert s.result() == src  # again, from pooled memory
    assert cr_lib.unified(src, b"\xff", b"") == src

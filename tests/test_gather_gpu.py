"""Regions of 2 KiB with a given number of matches, around the counts at which the output takes another
path, at every alignment of the output and with matches at both ends of a region."""
import numpy as np
import pytest

from cuda_replace_b200.cuda_replace_wrapper import Session

pytestmark = pytest.mark.gpu

REGION = 2048


def _regions(counts, L, seed):
    """One region per entry of counts, each with that many occurrences of 1, 2, ..., L in bytes from 128 up."""
    rng = np.random.default_rng(seed)
    out = rng.integers(128, 256, size=len(counts) * REGION, dtype=np.uint8)
    pat = np.arange(1, L + 1, dtype=np.uint8)
    for r, m in enumerate(counts):
        slots = rng.permutation(REGION // L)[:m]
        if m > 1:
            slots[:2] = (0, REGION // L - 1) if r % 2 else slots[:2]
        for s in set(slots.tolist()):
            out[r * REGION + s * L:r * REGION + s * L + L] = pat
    return out, pat.tobytes()


COUNTS = [2, 3, 4, 8, 9, 16, 17, 32, 33, 63, 64, 65, 1, 0, 24, 48]


@pytest.mark.parametrize("L", [1, 2, 3, 20, 31])
@pytest.mark.parametrize("R", [0, 1, 2, 5, 16, 17, 40, 64])
def test_small_inputs(cr_lib, L, R):
    if R == L:
        R += 1
    rep = bytes((11 * i + 3) & 0x7F for i in range(R))
    with Session(cr_lib, b"") as s:
        for seed in range(3):
            data, pat = _regions(COUNTS, L, seed)
            for cut in (0, 1, 7):  # the regions' outputs at other alignments, matches across their ends
                src = bytes(cut) + data.tobytes()
                s.reset(src)
                assert s.apply(pat, rep) == len(src.replace(pat, rep))
                assert s.result() == src.replace(pat, rep), (seed, cut)


@pytest.mark.parametrize("L,R", [(1, 2), (3, 1), (5, 0), (2, 17), (20, 40)])
def test_large_inputs(cr_lib, L, R):
    """Above the size from which the other kernel takes the input."""
    rep = bytes((11 * i + 3) & 0x7F for i in range(R))
    data, pat = _regions(COUNTS * 8, L, 5)
    src = data.tobytes() + b"\x80\x80\x80"
    src = src * ((66 << 20) // len(src))
    want = src.replace(pat, rep)
    with Session(cr_lib, src) as s:
        assert s.apply(pat, rep) == len(want)
        assert s.result() == want

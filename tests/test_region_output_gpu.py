"""Regions that mix literal bytes and replacements: every replacement length class, match densities
around the piece limit, whole and partial 2 KiB regions, equal lengths (written in place)."""
import numpy as np
import pytest

from cuda_replace_b200.cuda_replace_wrapper import Session

pytestmark = pytest.mark.gpu


def _text(n, pat, every, seed):
    """n filler bytes with the pattern planted about every `every` bytes (bytes of the pattern do not
    occur in the filler)."""
    rng = np.random.default_rng(seed)
    filler = np.array([b for b in range(256) if b not in pat], dtype=np.uint8)
    buf = bytearray(filler[rng.integers(0, len(filler), size=n)].tobytes())
    at = 0
    while at + len(pat) <= n:
        buf[at:at + len(pat)] = pat
        at += len(pat) + int(rng.integers(0, 2 * every + 1))
    return bytes(buf)


@pytest.mark.parametrize("rep_len", [0, 1, 2, 3, 4, 5, 8, 31, 32, 33, 64, 65, 256])
@pytest.mark.parametrize("pat", [b"q", b"qz", b"qzx", b"qqz", b"aba", b"qwertyui", b"x" + b"y" * 63, b"k" + b"l" * 79])
def test_mixed_regions(cr_lib, pat, rep_len):
    rep = bytes((7 * i + 1) & 0xFF for i in range(rep_len))
    with Session(cr_lib, b"") as s:
        for n, every in [(2047, 3), (2048, 500), (2049, 1), (16384 + 65, 430), (65536, 9), (65536 + 1, 0),
                         (3 * 65536 + 2048 * 5 + 77, 70), (200_003, 510), (300_000, 30)]:
            data = _text(n, pat, every, n + rep_len)
            s.reset(data)
            assert s.apply(pat, rep) == len(data.replace(pat, rep))
            assert s.result() == data.replace(pat, rep), (n, every)

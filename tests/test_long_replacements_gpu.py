"""How a region's output is written, by its matches and the replacement's length: pieces, chunks gathered,
bytes scattered in rounds or straight to memory. Regions of 0 to 2048 matches, lengths around every limit, in the
region kernel (small inputs) and in the super-tile kernel (above 64 MiB; above 8 MiB for short patterns that
overlap themselves)."""
import numpy as np
import pytest

from cuda_replace_b200.cuda_replace_wrapper import Session

pytestmark = pytest.mark.gpu

KiB, MiB = 1 << 10, 1 << 20
COUNTS = [0, 1, 2, 3, 15, 16, 17, 31, 33, 64, 100, 128, 199, 200, 201, 300, 2048]
A, B = b"\x80", b"\x81"
PATTERNS = [A, A + B, A + A, A + B + A, A * 5, A + b"\x82" * 30 + B, A * 40, A + b"\x82" * 62 + B, A + b"\x82" * 63 + B,
            A + b"\x82" * 298 + B]


def _planted(pat, seed):
    """A text with COUNTS matches (as many as fit) in regions of 2 KiB, each count in four regions."""
    rng = np.random.default_rng(seed)
    out = []
    for m in COUNTS * 4:
        region = rng.integers(97, 123, size=2048, dtype=np.uint8)
        m = min(m, 2048 // len(pat))
        slots = rng.permutation(2048 // len(pat))[:m]
        slack = 2048 - 2048 // len(pat) * len(pat)
        shift = int(rng.integers(0, slack + 1))
        for k in slots.tolist():
            region[shift + k * len(pat):shift + (k + 1) * len(pat)] = np.frombuffer(pat, dtype=np.uint8)
        out.append(region)
    text = np.concatenate(out)
    return np.roll(text, int(rng.integers(0, 4096)))  # (counts that straddle the kernel's regions too)


def _rep(R):
    return (bytes(range(33, 96)) * (R // 63 + 1))[:R]


def _lengths(pat, short):
    return sorted({5, 16, 17, 32, 33, 64, 65, 256, 257, 1024, 1025, len(pat)} - ({5, 16, 32, 33, 257, 1024} if short else set()))


@pytest.mark.parametrize("pat", PATTERNS, ids=len)
def test_region_kernel(cr_lib, pat):
    text = _planted(pat, len(pat)).tobytes()
    with Session(cr_lib, b"") as s:
        for R in _lengths(pat, False):
            rep = _rep(R)
            exp = text.replace(pat, rep)
            s.reset(text)
            assert s.apply(pat, rep) == len(exp)
            assert s.result() == exp, R


@pytest.mark.parametrize("pat", [p for p in PATTERNS if p not in (A * 5, A * 40)], ids=len)
def test_super_tile_kernel(cr_lib, pat):
    n = (8 if pat in (A + A, A + B + A) else 64) * MiB + 12345
    block = np.random.default_rng(3).integers(97, 123, size=2 * MiB, dtype=np.uint8)
    planted = _planted(pat, len(pat))
    block[777777:777777 + len(planted)] = planted
    text = np.resize(block, n)
    text[-len(planted):] = planted  # the last, partial super-tile too
    text = text.tobytes()
    with Session(cr_lib, b"") as s:
        for R in _lengths(pat, True):
            rep = _rep(R)
            exp = text.replace(pat, rep)
            s.reset(text)
            assert s.apply(pat, rep) == len(exp)
            assert s.result() == exp, R

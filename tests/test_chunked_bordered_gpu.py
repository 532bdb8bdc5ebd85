"""unified() above 256 MiB uploads, replaces and downloads in chunks of 32 MiB: patterns of 5 to 64 bytes that
overlap themselves, in runs across every chunk's end at many offsets and in a text that is one run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MiB = 1 << 20
CHUNK = 32 * MiB
PATTERNS = [b"a" * 5, b"ab" * 10, b"-" * 32, b"-" * 40, b"aba" * 17, b"a" * 64, b"ab" * 32, b"ab" + b"c" * 60 + b"ab"]


def _pinned(n):
    import torch
    t = torch.empty(n, dtype=torch.uint8, pin_memory=True)
    return t, t.numpy()


@pytest.fixture(scope="module")
def text():
    rng = np.random.default_rng(5)
    base = rng.integers(100, 122, size=MiB, dtype=np.uint8)
    n = 8 * CHUNK + 4321
    return _pinned(n)[1], np.resize(base, n)


@pytest.mark.parametrize("pat", PATTERNS)
@pytest.mark.parametrize("rep", [b"", b"<hr>", b"0123456789" * 8])
def test_runs_across_every_chunk_end(cr_lib, text, pat, rep):
    buf, base = text
    buf[:] = base
    L = len(pat)
    period = next(k for k in range(1, L) if pat[k:] == pat[:-k])
    rng = np.random.default_rng(L + len(rep))
    for end in range(CHUNK, len(buf), CHUNK):
        run = pat[:period] * int(rng.integers(2, 400))  # from a few bytes to beyond a region
        run += run[:int(rng.integers(0, period + 1))]
        at = end - int(rng.integers(0, len(run) + 2 * L))
        run = run[:len(buf) - at]
        buf[at:at + len(run)] = np.frombuffer(run, dtype=np.uint8)
    src = buf.tobytes()
    exp = src.replace(pat, rep)
    assert cr_lib.unified(src, pat, rep) == exp  # pageable
    if rep:
        assert cr_lib.unified(buf, pat, rep) == exp  # page-locked


@pytest.mark.parametrize("L,R", [(5, 3), (31, 1), (33, 40), (64, 65)])
def test_one_run(cr_lib, text, L, R):
    buf, _ = text
    buf[:] = ord("a")
    buf[3 * CHUNK - 7] = ord("b")
    src = buf.tobytes()
    pat, rep = b"a" * L, (b"0123456789" * 7)[:R]
    exp = src.replace(pat, rep)
    assert cr_lib.unified(src, pat, rep) == exp
    assert cr_lib.unified(buf, pat, rep) == exp

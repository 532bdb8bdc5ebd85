"""The super-tile kernel on one apply: inputs above the line to the region kernel (64 MiB; 16 MiB for free patterns
of more than 64 bytes; 8 MiB for short patterns that overlap themselves), ends inside a super-tile,
query_prefix, the presence index, seeded applies."""
import bisect
import re

import numpy as np
import pytest

from cuda_replace_b200.cuda_replace_wrapper import Session

pytestmark = pytest.mark.gpu

MiB = 1 << 20
A, B = b"\x80", b"\x81"
FREE65, FREE300 = A + b"\x82" * 63 + B, A + b"\x82" * 298 + B
CASES = [(A, 64), (A + B, 64), (A + b"\x82" * 60 + B, 64), (FREE65, 16), (FREE300, 16), (A + A, 8), (A + B + A, 8),
         (A + B + A + B, 8)]


def _text(pat, n):
    """Sparse matches at irregular distances; a run of the pattern at the end."""
    rng = np.random.default_rng(len(pat))
    block = rng.integers(97, 123, size=3 * MiB + 4321, dtype=np.uint8)
    at = 0
    while at + len(pat) < len(block):
        block[at:at + len(pat)] = np.frombuffer(pat, dtype=np.uint8)
        at += int(rng.integers(len(pat), 9000))
    out = np.resize(block, n)
    out[-5 * len(pat):] = np.frombuffer(pat * 5, dtype=np.uint8)
    return out.tobytes()


@pytest.mark.parametrize("pat,line", CASES, ids=lambda v: str(len(v)) if isinstance(v, bytes) else "")
@pytest.mark.parametrize("past", [0, 1, 65536 + 2047])
def test_result_and_query_prefix(cr_lib, pat, line, past):
    n = line * MiB + past
    text = _text(pat, n)
    starts = [m.start() for m in re.finditer(re.escape(pat), text)]  # leftmost, not overlapping
    with Session(cr_lib, text) as s:
        for rep in (b"", b"<>", pat[::-1]):
            s.reset(text)
            s.apply(pat, rep)
            assert s.result() == text.replace(pat, rep)
        assert s.stats()[0] == len(starts)
        for limit in (0, 1, 2048, 16384, 24575, 49153, 65536, n // 2 + 7, n - len(pat), n - 1, n):
            k = bisect.bisect_left(starts, limit)
            assert s.query_prefix(limit) == (k, starts[k - 1] if k else -1), limit


@pytest.mark.parametrize("pat,line", CASES, ids=lambda v: str(len(v)) if isinstance(v, bytes) else "")
def test_index_and_seeded(cr_lib, pat, line):
    n = line * MiB + 777
    text = bytearray(_text(pat, n))
    text[2 * MiB:5 * MiB] = b"k" * (3 * MiB)  # chunks without the pattern's first byte
    text = bytes(text)
    with Session(cr_lib, text) as s:
        s.build_index()
        s.apply(pat, b"#")
        assert s.result() == text.replace(pat, b"#")
        s.reset(text)
        _, last = s.apply_seeded(pat, b"#", 12345 - len(pat))  # no match may start before 12345
        exp = text[:12345] + text[12345:].replace(pat, b"#")
        assert s.result() == exp
        i, want = text.find(pat, 12345), -1
        while i != -1:
            want, i = i, text.find(pat, i + len(pat))
        assert last == want

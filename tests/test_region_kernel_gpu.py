"""The region kernel and the line between it and the super-tile kernel: sizes around its 2 KiB regions
and its super-tiles (24 KiB, 48 KiB for patterns that overlap themselves), patterns of every carry class, uniform and periodic texts, query_prefix."""
import numpy as np
import pytest

from cuda_replace_b200.cuda_replace_wrapper import Session

pytestmark = pytest.mark.gpu

T = 49152
SIZES = [1, 63, 64, 65, 2047, 2048, 2049, T // 2 - 1, T // 2, T // 2 + 1, T - 1, T, T + 1, T + 2048, 2 * T + 2049,
         7 * T + 31, 200 * T + 777]
PATTERNS = [b"a", b"aa", b"aaa", b"aaaa", b"aaaaa", b"a" * 31, b"a" * 32, b"a" * 33, b"a" * 40, b"a" * 63, b"a" * 64,
            b"ab", b"aba", b"abab", b"ababa", b"abaababaab", b"ab" * 16, b"ab" * 20 + b"a", b"abc" * 21,
            b"ba", b"baaa", b"b" + b"a" * 63, b"ab" + b"c" * 62 + b"ab"]


def _texts(n, seed):
    rng = np.random.default_rng(seed)
    yield b"a" * n
    yield (b"ab" * (n // 2 + 1))[:n]
    yield np.frombuffer(b"ab", dtype=np.uint8)[(rng.random(n) < 0.1).astype(int)].tobytes()
    yield np.frombuffer(b"abc", dtype=np.uint8)[rng.integers(0, 3, size=n)].tobytes()


@pytest.mark.parametrize("pat", PATTERNS)
def test_sizes_and_carries(cr_lib, pat):
    with Session(cr_lib, b"") as s:
        for n in SIZES:
            for i, data in enumerate(_texts(n, n)):
                rep = (b"", b"XY", b"Z" * len(pat), b"0123456789" * 5)[i]
                exp = data.replace(pat, rep)
                s.reset(data)
                assert s.apply(pat, rep) == len(exp)
                assert s.result() == exp, (n, i)
                if len(pat) <= n <= 8 * T:
                    for limit in {0, 1, n // 2, n - 1, n, min(n, T), min(n, 2048)}:
                        kept, last, q = 0, -1, data.find(pat)
                        while q != -1 and q < limit:
                            kept, last = kept + 1, q
                            q = data.find(pat, q + len(pat))
                        assert s.query_prefix(limit) == (kept, last), (n, i, limit)


@pytest.mark.parametrize("pat,edge", [(b"q", 64 << 20), (b"qz", 64 << 20), (b"qq", 8 << 20)])
def test_either_side_of_the_kernel_choice(cr_lib, pat, edge):
    rng = np.random.default_rng(len(pat))
    base = rng.integers(0, 256, size=edge + 1, dtype=np.uint8)
    base[:: 4099] = pat[0]
    base[1:: 4099] = pat[-1]
    data = base.tobytes()
    with Session(cr_lib, b"") as s:
        for n in (edge - 1, edge, edge + 1):
            s.reset(data[:n])
            s.apply(pat, b"#..#")
            assert s.result() == data[:n].replace(pat, b"#..#")

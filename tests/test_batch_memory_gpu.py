"""Device memory of apply_batch with its lengths chained on the device: look-back tables linear in the
input, and one apply per pair where the chain's worst case does not fit."""
import pytest

from cuda_replace_b200.cuda_replace_wrapper import Session

pytestmark = pytest.mark.gpu

MiB = 1 << 20


def _free():
    import torch
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("pat", [b"a" * 5, b"xy" * 10, b"-" * 32, b"-" * 40, b"ab" * 32])
def test_tables_grow_with_the_input_only(cr_lib, pat):
    src = (b"The quick brown fox " * 50 + pat + pat[:-1] + b" ") * ((160 * MiB) // (1000 + 2 * len(pat)))
    pairs = [(pat, b"<hr>"), (b"fox", b"dog")]
    with Session(cr_lib, src) as s:
        before = _free()
        s.apply_batch(pairs)
        taken = before - _free()
        exp = src
        for p, r in pairs:
            exp = exp.replace(p, r)
        assert s.result() == exp
    # the second buffer (with its headroom) and scratch: 16 KiB tiles of 64 entries are n / 32
    assert taken < len(src) + len(src) // 4 + len(src) // 16 + 64 * MiB, taken


def test_worst_case_beyond_memory_goes_pair_by_pair(cr_lib):
    import torch

    n = 256 * MiB
    line = b"." * 997 + b"-" * 40
    src = (line * (n // len(line) + 1))[:n]
    pairs = [(b"-" * 40, b"=" * 159), (b"==.", b"#")]  # the first may take the length to 4 n: two such buffers
    with Session(cr_lib, src) as s:
        torch.cuda.empty_cache()
        ballast = torch.empty(_free() - 1700 * MiB, dtype=torch.uint8, device="cuda")
        try:
            s.apply_batch(pairs)
            got = s.result()
        finally:
            del ballast
            torch.cuda.empty_cache()
        assert got == src.replace(*pairs[0]).replace(*pairs[1])

"""Device memory that finished streams keep for the next one goes back when something else needs it."""
import pytest

from cuda_replace_b200.cuda_replace_wrapper import Server, Session, gpu_replace_streaming

pytestmark = pytest.mark.gpu

MiB = 1 << 20


def _free():
    import torch
    return torch.cuda.mem_get_info()[0]


@pytest.fixture
def little_memory(cr_lib):
    """A device with idle stream blocks and, apart from them, 48 MiB."""
    import torch

    cr_lib.lib.cuda_replace_jobs_release()
    src = b"no match in any of this " * (6 * MiB)
    before = _free()
    assert gpu_replace_streaming(cr_lib, src, [(b"~", b"!"), (b"^", b"!")], 32 * MiB) == src
    assert before - _free() > 128 * MiB  # kept
    torch.cuda.empty_cache()
    ballast = torch.empty(_free() - 48 * MiB, dtype=torch.uint8, device="cuda")
    yield
    del ballast
    torch.cuda.empty_cache()


def test_server_opens(cr_lib, little_memory):
    with Server(cr_lib, hbm_budget=96 * MiB, max_jobs_per_batch=8) as srv:
        t = srv.submit(b"abcabc" * 1000, [(b"bc", b"x")])
        assert srv.wait(t) == b"axax" * 1000


def test_apply_tables_fit(cr_lib):
    """The look-back tables of a long pattern that overlaps itself: 8 bytes x L for every 16 KiB."""
    import torch

    pat = b"ab" * 1024
    src = b"-" * 777 + pat * 3 + b"cd" * (16 * MiB) + pat
    with Session(cr_lib, src) as s:
        assert s.apply(b"~", b"!") == len(src)  # both buffers
        cr_lib.lib.cuda_replace_jobs_release()
        big = b"no match in any of this " * (6 * MiB)
        assert gpu_replace_streaming(cr_lib, big, [(b"~", b"!"), (b"^", b"!")], 32 * MiB) == big
        torch.cuda.empty_cache()
        ballast = torch.empty(_free() - 16 * MiB, dtype=torch.uint8, device="cuda")
        try:
            s.apply(pat, b"Q")
            assert s.result() == src.replace(pat, b"Q")
        finally:
            del ballast
            torch.cuda.empty_cache()


def test_release_gives_them_back(cr_lib):
    src = b"no match in any of this " * (6 * MiB)
    assert gpu_replace_streaming(cr_lib, src, [(b"~", b"!"), (b"^", b"!")], 32 * MiB) == src
    before = _free()
    cr_lib.lib.cuda_replace_jobs_release()
    assert _free() - before > 128 * MiB

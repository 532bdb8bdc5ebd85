"""A new session knows nothing of the results of one that was closed before it, although it may be given
the same page-locked memory."""
import pytest

from cuda_replace_b200.cuda_replace_wrapper import Session

pytestmark = pytest.mark.gpu


def test_new_session_after_an_overflow(cr_lib):
    src = b"a" * (4 << 20)
    for _ in range(3):
        with Session(cr_lib, src) as s:
            assert s.apply(b"a", b"b" * 100) == 100 * len(src)  # outgrows its first buffer
        with Session(cr_lib, b"x,z" * 1000) as s:  # its first launches bear the same numbers
            s.apply_batch([(b"x", b"yy"), (b"z", b"w")])
            assert s.result() == b"yy,w" * 1000

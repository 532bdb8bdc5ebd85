"""The presence index outlives a batch whose stage tables have to grow: the index belongs to the
session, and a later build_index writes into the same memory."""
import pytest

from cuda_replace_b200 import workloads as WL

from cuda_replace_b200 import cuda_replace_wrapper as Wr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs", [4, 64])
def test_index_then_growing_batch_then_index(cr_lib, pairs):
    src = WL.text_corpus((3 << 20) + 77, seed=5) + b"<01><07>" * 100
    rules = [(b"<%02d>" % k, b"[%d]" % k) for k in range(pairs)]
    more = [(b"[%d]" % k, b"<<%02d>>" % k) for k in range(pairs)] + rules * 2
    with Wr.Session(cr_lib, src) as s:
        want = src
        for batch in (rules, more):
            s.build_index(16384)
            s.apply_batch(batch)
            for a, b in batch:
                want = want.replace(a, b)
            assert s.result() == want
        s.build_index(16384)
        s.apply(b"e", b"EE")
        assert s.result() == want.replace(b"e", b"EE")

"""What the binding refuses before it calls the library (no library call is made here). CPU only."""
import ctypes as C

import pytest

from cuda_replace_b200 import cuda_replace_wrapper as Wr

ASYNC = C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_void_p, C.c_size_t, C.c_char_p, C.c_int, C.c_char_p, C.c_int, C.c_void_p,
                    C.c_size_t, C.c_void_p)


@pytest.fixture
def calls(fake_lib_path):
    lib, seen = Wr.CudaReplaceLib(fake_lib_path), []
    lib._async = ASYNC(lambda *a: seen.append(a) or 0)
    return lib, seen


@pytest.mark.parametrize("bad", [b"bytes", "text", 1.5, (C.c_uint8 * 16)(), C.c_char_p(b"x"), [16]])
@pytest.mark.parametrize("where", ["d_in", "d_out", "stream", "n", "out_cap"])
def test_device_addresses_are_integers(calls, bad, where):
    lib, seen = calls
    with Wr.Session(lib, b"") as s:
        args = dict(d_in=4096, n=16, pat=b"a", rep=b"b", d_out=8192, out_cap=64, stream=0)
        s.apply_device_async(**args)
        assert seen.pop()[1:] == (4096, 16, b"a", 1, b"b", 1, 8192, 64, None)
        with pytest.raises(TypeError):
            s.apply_device_async(**{**args, where: bad})
    assert not seen


@pytest.mark.parametrize("bad", ["text", bytearray(b"ab"), memoryview(b"ab"), 5, None])
def test_patterns_are_bytes(calls, bad):
    lib, seen = calls
    with Wr.Session(lib, b"abc") as s:
        for pat, rep in ((bad, b"x"), (b"x", bad)):
            for call in (lambda: s.apply_device_async(4096, 16, pat, rep, 8192, 64), lambda: s.apply(pat, rep),
                         lambda: lib.unified(b"abc", pat, rep)):
                with pytest.raises(TypeError):
                    call()
    assert not seen


def test_result_of_a_closed_session_names_the_call(fake_lib_path):
    s = Wr.Session(Wr.CudaReplaceLib(fake_lib_path), b"abc")
    s.close()
    with pytest.raises(RuntimeError, match="cuda_replace_result failed"):
        s.result()

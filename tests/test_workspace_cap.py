"""While a cap on the serve loop's memory is set, nothing that the cap does not
count stays allocated between standalone calls (tests/harness/workspace.cpp,
the library's workspace over an allocator of fixed size)."""
import ctypes as C

from test_workspace_memory import MB, lib  # noqa: F401 -- the fixture


def test_nothing_is_kept_under_a_cap(lib):  # noqa: F811
    lib.ws_cap.argtypes, lib.ws_cap.restype = [C.c_void_p, C.c_int], None
    lib.ws_cap_during_call.argtypes, lib.ws_cap_during_call.restype = [C.c_void_p, C.c_size_t], C.c_size_t
    w = lib.ws_open(200 * MB)
    assert lib.ws_call(w, 3 * MB, 0) == 1 and lib.ws_used() == 4 * MB
    lib.ws_cap(w, 1)
    assert lib.ws_used() == 0
    assert lib.ws_call(w, 3 * MB, 5 * MB) == 1 and lib.ws_used() == 0
    lib.ws_cap(w, 0)
    assert lib.ws_call(w, 3 * MB, 0) == 1 and lib.ws_used() == 4 * MB
    assert lib.ws_cap_during_call(w, 8 * MB) == 0
    assert lib.ws_close(w) == 0

"""The query calls of the Python mirror, with the compiled helper and without: the same arrays reach the
C ABI, the same decisions come back, and the same arguments are refused."""
import ctypes as C

import pytest


@pytest.fixture(scope="module")
def ways(built_extension):
    from morello_b200 import _lib, build
    out = [_lib.call_many_in_python]
    if build._has_python_headers():
        out.append(_lib.call_many())
        assert out[1] is not out[0]
    return out


def _answers(ways, blobs, limits, status=0):
    """Per way of calling: what the function was called with, and what the caller got."""
    from morello_b200 import _lib
    from morello_b200.db import Decision
    got = []
    for call in ways:
        seen = []

        @C.CFUNCTYPE(C.c_int, C.c_void_p, C.POINTER(C.c_uint8), C.POINTER(C.c_uint64), C.c_size_t, C.POINTER(C.c_uint64), C.POINTER(_lib.Decision))
        def fake(ctx, data, off, n, lim, out):
            offs = off[:n + 1]
            seen.append((ctx, bytes(data[:offs[n]]), offs, lim[:4 * n]))
            for i in range(n):
                out[i].found = (1, 0, -1)[i % 3]
                out[i].action, out[i].main_cost, out[i].depth = 60000 + i, 0xFFFFFFFF - i, 255
                for k in range(4):
                    out[i].peaks[k] = (1 << 40) + k
            return status

        try:
            res = call(C.cast(fake, C.c_void_p).value, 0x1234, blobs() if callable(blobs) else blobs, limits() if callable(limits) else limits, Decision)
        except Exception as e:
            res = type(e)
        got.append((seen, res))
    return got


class _Index:
    def __index__(self):
        return 7


@pytest.mark.parametrize("blobs,limits", [
    ([], []),
    ([b"ab", b"", b"cdefg"], [(1, 2, 3, 4), [5, 6, 7, 8], (0, 0, 1 << 63, (1 << 64) - 1)]),
    ((bytearray(b"xy"), memoryview(b"z1")), ([1, 2, 3, 4, 5], (-1, 0, 1, 2))),        # longer limits, a negative number
    ([b"ab"] * 7, [(1, 2, 3, 4)] * 3),                                                # the rest at zero
    ([b"ab", b"cd"], lambda: (iter((k, k, k, k)) for k in range(2))),
    ([b"ab"], [(_Index(), True, 0, 2)]),
])
def test_the_same_call(ways, blobs, limits):
    got = _answers(ways, blobs, limits)
    for seen, res in got:
        assert len(seen) == 1 and res[0] == 0
        assert (seen, res) == got[0]
        assert all((d.action, d.peaks) == (0, (0, 0, 0, 0)) for d in res[1] if d.found != 1)
    assert all(res == (-7, None) for _, res in _answers(ways, blobs, limits, status=-7))


@pytest.mark.parametrize("blobs,limits,error", [
    ([b"ab"], [(1, 2, 3, 4)] * 2, IndexError),
    ([b"ab"], [(1, 2, 3)], IndexError),
    ([b"ab"], [(1, 2.0, 3, 4)], TypeError),
    ([b"ab"], [5], TypeError),
    ([3], [(1, 2, 3, 4)], TypeError),
])
def test_the_same_refusals(ways, blobs, limits, error):
    for seen, res in _answers(ways, blobs, limits):
        assert not seen and issubclass(res, error)


def test_the_helper_of_another_interpreter_is_not_taken(built_extension):
    import sysconfig
    from morello_b200 import build
    assert build.PYHOST_PATH.endswith(sysconfig.get_config_var("EXT_SUFFIX"))

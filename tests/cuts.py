"""How a call is cut (awq_b200_gemm_cut), for tests that name the cut they are for."""
import collections
import ctypes

# clusters of i CTAs that a B200 holds at once, one CTA per SM; which sizes above 8 fit how often differs by GPU
B200 = [0, 148, 74, 45, 33, 26, 22, 15, 15, 15, 11, 7, 7, 7, 7, 7, 7]

Cut = collections.namedtuple("Cut", "kernel tokens chunk cluster tiles accumulators")


def cut(m, k, n, group, kernel=0, room=None):
    """Of a call with its scratch; `room` as B200 above, None: of the current device."""
    from awq_b200 import _lib
    told = (ctypes.c_int * 6)(*[-1] * 6)
    rc = _lib.load().awq_b200_gemm_cut(m, n, k, group, kernel, (ctypes.c_int * 17)(*room) if room else None, told)
    assert rc == 0, rc
    return Cut(*told)

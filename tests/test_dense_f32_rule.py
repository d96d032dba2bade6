"""Which calls the tiles of dense f32 attention take, decided on the host."""
import ctypes

import pytest

from singe_b200 import kernel_sys as ks

P, I, L, F = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float


class DenseF32(ctypes.Structure):      # csrc/attention_f32.cuh
    _fields_ = ([(name, P) for name in ("query", "out", "lse", "key", "value", "sinks")]
                + [(name, I) for name in ("heads", "kv_heads", "query_len", "key_len", "head_dim", "causal")]
                + [(name, L) for name in ("window", "q_batch", "q_head", "q_row", "k_batch", "k_head", "k_row")]
                + [("scale", F), ("softcap", F)])


def takes(**changes):
    call = dict(query=64, out=64, key=64, value=64, heads=1, kv_heads=1, query_len=16, key_len=64, head_dim=4, window=0)
    call.update(changes)
    function = getattr(ks.lib(), "_ZN5singe25dense_attention_f32_takesERKNS_8DenseF32Em")
    function.argtypes, function.restype = [ctypes.POINTER(DenseF32), ctypes.c_size_t], ctypes.c_bool
    return function(ctypes.byref(DenseF32(**call)), 1)


@pytest.mark.parametrize("name", ["query_len", "key_len"])
def test_positions_stay_below_2_31(name):
    # four teams of 64 keys step over each other, and the last tile's keys lie behind the last step
    most = 2 ** 31 - 1 - 5 * 64
    assert takes(**{name: most})
    assert not any(takes(**{name: length}) for length in range(most + 1, 2 ** 31))


def test_other_limits():
    assert takes() and takes(head_dim=128)
    assert not any(takes(**change) for change in (dict(head_dim=6), dict(head_dim=132), dict(query_len=15), dict(query=68),
                                                  dict(out=72), dict(key=4), dict(value=8)))

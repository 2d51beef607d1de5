"""Rules by which calls are routed to kernels and the arguments that launches get, as far as the host decides them: no GPU."""
import ctypes as C

import pytest
import torch

from ollama_b200.ops import cuda as K


@pytest.mark.parametrize("hd", [64, 128])
def test_int8_caches_whose_scales_are_not_aligned_go_to_the_scalar_decode_kernel(hd):
    """The ring of the tensor-core kernel copies the hd / 16 bytes of a row's scales at once; other bases are read one scale after the other.  (Only addresses are looked at.)"""
    base = 1 << 20

    def takes(k_off, v_off, scales=True, heads=8):
        a = K.AttnDecodeArgs(base, base, base, base, base, heads, 2, 256, 1, 1.0, 0.0, 0, base, base, base + k_off if scales else None, base + v_off if scales else None)
        return K.lib().b2_attn_decode_mma_takes(C.byref(a), hd)

    for off in range(0, 16, 2):
        whole = off % (hd // 16) == 0
        assert takes(off, 0) == takes(0, off) == takes(off, off) == int(whole), off
    assert takes(0, 0, scales=False) == 1
    assert takes(0, 0, heads=7) == 0 and takes(0, 0, heads=64) == 0

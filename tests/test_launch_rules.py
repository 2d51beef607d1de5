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


def test_depth_of_decode_attention_by_the_ctas_an_sm_gets():
    """148 SMs, 8 KV heads, 16 splits: four stages up to one CTA an SM, int8 caches too; three up to two; else as few as there are."""
    def depth(nb, q8, n_splits=16, n_ctx=8192):
        at = 1 << 20
        return K.lib().b2_attn_decode_depth(C.byref(K.AttnDecodeArgs(at, at, at, at, at, 32, 8, n_ctx, n_splits, 1.0, 0.0, 0, at, at, *([at, at] if q8 else [None, None]))), nb)

    assert [depth(nb, False) for nb in (1, 2, 3, 8)] == [4, 3, 2, 2]
    assert [depth(nb, True) for nb in (1, 2, 3, 8)] == [4, 3, 3, 3]
    assert depth(1, False, n_splits=4, n_ctx=500) == 2 and depth(1, True, n_splits=4, n_ctx=500) == 3
    for forced in (2, 3, 4):
        K.attn_decode_stages(forced)
        try:
            assert [depth(nb, False) for nb in (1, 8)] == [forced] * 2 and [depth(nb, True) for nb in (1, 8)] == [max(3, forced)] * 2
        finally:
            K.attn_decode_stages(0)


def test_expert_rows_are_not_laid_out_for_chunks_that_no_kernel_takes():
    for chunk in (0, 4, 12, 40, 56, 128):
        with pytest.raises(ValueError):
            K.MoeFp4(8, 4, 64, 64, "cpu", chunk)
    assert all(K.moe_fp4_chunk(rows / 4) in K.MoeFp4.CHUNKS for rows in range(1, 400))


class Launches:
    """Stands for the kernel library: keeps the arguments of each call."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        class Entry:
            def __call__(_, *args):
                self.calls.append((name, args))
                return 0
        return Entry()


@pytest.fixture
def launches(monkeypatch):
    got = Launches()
    monkeypatch.setattr(K, "lib", lambda: got)
    monkeypatch.setattr(K, "stream", lambda: None)
    monkeypatch.setattr(K, "gemm_bf16_scratch", lambda *_: 0)
    return got


@pytest.mark.parametrize("call,at", [(K.gemm_bf16, 9), (K.gemm_bf16_out16, 8), (lambda a, b, pdl: K.gemm_bf16_glu(a, b, "silu", pdl=pdl), 11)])
def test_a_matrix_that_is_copied_for_the_product_is_not_fetched_early(launches, call, at):
    """pdl 2 says that b does not depend on the kernel just before; where the wrapper copies b, that kernel is the copy."""
    a, b = torch.zeros(4, 64, dtype=torch.bfloat16), torch.zeros(32, 64, dtype=torch.bfloat16)
    strided, turned = torch.zeros(32, 128, dtype=torch.bfloat16)[:, :64], torch.zeros(64, 32, dtype=torch.bfloat16).t()
    for m, pdl, want in ((b, 2, 2), (b, 0, 0), (strided, 2, 1), (turned, 2, 1), (strided, 1, 1), (strided, 0, 0)):
        call(a, m, pdl=pdl)
        assert launches.calls[-1][1][at] == want, (want, launches.calls[-1])


@pytest.mark.parametrize("pdl", [False, True])
def test_products_of_stack_models_follow_the_engines_overlap_flag(monkeypatch, pdl):
    from types import SimpleNamespace as NS

    from ollama_b200.engine.blocks import Step
    from ollama_b200.engine.stack import StackBackend
    from ollama_b200.ops import rows as O
    got = []
    monkeypatch.setattr(O, "_call", lambda name, g, *_: got.append((name, g.pdl)))
    monkeypatch.setattr(O, "_split_floats", lambda *_: 0)
    h, w, out = torch.zeros(40, 64, dtype=torch.bfloat16), torch.zeros(32, 64, dtype=torch.bfloat16), torch.zeros(40, 32)
    O.gemm(h, w, out)
    assert got.pop() == ("b2_gemm_rows", 1)
    O.gemm(h, w, out, pdl=pdl)
    StackBackend._mm(NS(pdl=pdl, _n=0), h, w, out)
    step = NS(small=False, be=NS(pdl=pdl), m=NS(tokens=None), launched=lambda: None)
    Step.product(step, h, NS(w=w, bias=None), out)
    Step.enter(step, h, NS(w=w, bias=None), out)
    assert got == [("b2_gemm_rows", int(pdl))] * 4


@pytest.mark.parametrize("segs", [[(0, [5] * 9, 56)], [(0, [5], 64)], [(2, [5], 0)], [(-1, [5], 0)], [(0, [5], -1)], [(0, [5] * 4, 0), (1, [5] * 40, 25)]])
def test_prompt_rows_outside_the_cache_are_refused_before_a_launch(launches, segs):
    """The cache append writes at slot and position as they come; attention, which looks at the length, follows it."""
    from types import SimpleNamespace as NS

    from ollama_b200.engine.b200 import B200Backend
    be = NS(n_slots=2, n_ctx=64, cfg=NS(), device="cpu")
    with pytest.raises(ValueError):
        B200Backend._forward_rows(be, segs)
    assert not launches.calls

"""Binding of the prompt pass (kernels/prefill_pass.cu): all launches of a run of dense layers from one native call."""
from __future__ import annotations

import ctypes as C

import torch

from . import cuda as K
from . import sk as SK

P, I, F = C.c_void_p, C.c_int, C.c_float


class PassLayer(C.Structure):
    _fields_ = [("attn_norm", P), ("ffn_norm", P), ("wqkv", P), ("wo", P), ("gu", P), ("down", P), ("bqkv", P), ("bo", P), ("bgu", P), ("bdown", P), ("units", SK.SgSeg * 6),
                ("q_norm", P), ("k_norm", P), ("sinks", P), ("inv_freq", P), ("mscale", F), ("window", I), ("k_cache", P), ("v_cache", P), ("k_scale", P), ("v_scale", P)]


class PassSeg(C.Structure):
    _fields_ = [("row0", I), ("rows", I), ("slot", I), ("pos0", I)]


class PassArgs(C.Structure):
    _fields_ = [("rows", I), ("d", I), ("n_heads", I), ("n_kv_heads", I), ("hd", I), ("n_rot", I), ("neox", I), ("n_ctx", I), ("n_slots", I), ("ff", I), ("causal", I), ("act", I),
                ("eps", F), ("scale", F), ("softcap", F), ("alpha", F), ("limit", F), ("positions", P), ("slots", P), ("x", P), ("qkv", P), ("q", P), ("o", P), ("h", P), ("f", P),
                ("x16", P), ("ws", P), ("ws_floats", C.c_longlong), ("status", P), ("units", I), ("tc", I), ("pdl", I), ("kv16", P), ("kv16_halves", C.c_longlong), ("launches", I)]


class PromptPass:
    """The layers of an engine (the ``be`` of its methods) with their caches, as :func:`run` hands them to the native pass.  ``wide``: every layer has resident 16-bit matrices; ``units``: unit-ordered
    ones.  Holds addresses of the engine's tensors, which it keeps alive, and nothing of a call."""

    def __init__(self, be):
        c = be.cfg
        self.layers = (PassLayer * len(be.layers))()
        self.wide = self.units = True
        self.keep = []
        for i, (L, a) in enumerate(zip(be.layers, self.layers)):
            local = L.swa and c.rope_base_local > 0
            b16 = [L.wqkv16] + [getattr(w, "bf16", None) for w in (L.wo, L.gu, L.down)]
            bias = [L.bqkv, L.wo.bias, L.gu.bias, L.down.bias]
            self.wide &= all(w is not None and w.shape[1] % 8 == 0 for w in b16)
            self.units &= L.sk is not None
            ts = [L.attn_norm, L.ffn_norm, *b16, *bias, L.q_norm, L.k_norm, L.sinks, be.inv_freq_local if local else be.inv_freq]
            a.attn_norm, a.ffn_norm, a.wqkv, a.wo, a.gu, a.down, a.bqkv, a.bo, a.bgu, a.bdown, a.q_norm, a.k_norm, a.sinks, a.inv_freq = map(K.ptr, ts)
            if L.sk is not None:
                for s, w in zip(a.units, [*L.sk.qkv, L.sk.o, L.sk.gu, L.sk.down]):
                    s.w, s.bias, s.type, s.n = w.units.data_ptr(), K.ptr(w.bias), w.wtype, w.n
                    ts += [w.units, w.bias]
            a.mscale, a.window = (1.0 if local else be.mscale), (c.sliding_window if L.swa else 0)
            a.k_cache, a.v_cache, a.k_scale, a.v_scale = map(K.ptr, (be.k_cache[i], be.v_cache[i], be.k_scale[i], be.v_scale[i]))
            self.keep += [ts, be.k_cache[i], be.v_cache[i], be.k_scale[i], be.v_scale[i]]
        self.windows = {a.window for a in self.layers}
        self.ws = SK.Workspace(be.device) if self.units else None

    def run(self, be, x: torch.Tensor, positions: torch.Tensor, slots: torch.Tensor, segs: list[tuple[int, int, int, int]], units: bool, tc: bool) -> int:
        """The layers on the residual rows ``x`` (fp32 [rows, d], in place).  ``segs``: (first row, rows, slot, first position) of each sequence.  Returns the launches."""
        c, dev, n = be.cfg, x.device, x.shape[0]

        def rows(cols, dtype=torch.float32):
            return torch.empty(n, cols, device=dev, dtype=dtype)

        qkv, q, o = rows((c.n_heads + 2 * c.n_kv_heads) * c.head_dim), rows(c.q_dim), rows(c.q_dim, torch.bfloat16)
        h = None if units else rows(c.d_model, torch.bfloat16)
        f = rows(c.d_ff, torch.float32 if units else torch.bfloat16)
        x16 = torch.empty(SK.rows16_bytes(min(n, SK.ROWS16_MAX), max(c.d_model, c.q_dim, c.d_ff)), device=dev, dtype=torch.uint8) if units else None
        ws = self.ws if units else None
        size = 0 if units else max(K.gemm_bf16_scratch(n, *nk) for nk in (((c.n_heads + 2 * c.n_kv_heads) * c.head_dim, c.d_model), (c.d_model, c.q_dim), (c.d_model, c.d_ff)))
        parts = torch.empty(size, device=dev, dtype=torch.float32) if size else None
        q8 = tc and c.head_dim in (64, 128) and be.k_scale[0] is not None and max(p0 + r for _, r, _, p0 in segs) > 64
        kv16 = None
        if q8:
            head = max(K.attn_prefill_q8_head(p0, p0 + r, w, c.head_dim) for _, r, _, p0 in segs for w in self.windows)
            kv16 = K.attn_prefill_q8_scratch(head, c.n_kv_heads, dev)
        a = PassArgs(n, c.d_model, c.n_heads, c.n_kv_heads, c.head_dim, c.rope_dim, int(c.rope_style == "neox"), be.n_ctx, be.n_slots, c.d_ff, int(c.causal), K._ACT[c.act],
                     c.norm_eps, be.attn_scale, c.attn_softcap, c.swiglu_alpha, c.swiglu_limit, K.ptr(positions), K.ptr(slots), K.ptr(x), K.ptr(qkv), K.ptr(q), K.ptr(o), K.ptr(h),
                     K.ptr(f), K.ptr(x16), *((K.ptr(ws.ws), 0, K.ptr(ws.status)) if units else (K.ptr(parts), size, None)), int(units), int(tc),
                     int(be.pdl), K.ptr(kv16), kv16.numel() if kv16 is not None else 0, 0)
        sg = (PassSeg * len(segs))(*[PassSeg(*s) for s in segs])
        fn = K.lib().b2_prefill_pass
        fn.argtypes = [P, I, P, P, I, P]
        K._check(fn(self.layers, len(self.layers), C.byref(a), sg, len(segs), K.stream()), "prefill_pass")
        return a.launches

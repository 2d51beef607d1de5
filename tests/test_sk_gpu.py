"""The streaming tensor-core decode GEMV (kernels/gemv_sk.cu) against plain PyTorch fp32 statements."""
import pytest
import torch

from ollama_b200.gguf.types import GGMLType
from ollama_b200.models.weights import QWeight
from ollama_b200.ops import reference as R

pytestmark = pytest.mark.gpu


def _mods():
    from ollama_b200.ops import cuda as K
    from ollama_b200.ops import sk
    return K, sk


def _qw(t, n, k, seed):
    g = torch.Generator().manual_seed(seed)
    return QWeight.from_float("w", torch.randn(n, k, generator=g) * 0.05, t)


def _quant256_ref(x):
    """int8 with one scale per 256 elements, as the kernels quantise activations; returns the de-quantised values."""
    xb = x.view(x.shape[0], -1, 256)
    amax = xb.abs().amax(-1, keepdim=True)
    inv = torch.where(amax > 0, 127.0 / amax.clamp_min(1e-30), torch.zeros_like(amax))
    return (torch.round(xb * inv) * (amax / 127.0)).view_as(x)


def _close(y, ref, tol=2e-3):
    return torch.allclose(y, ref, atol=tol * ref.abs().max().item(), rtol=1e-3)


def test_quant256_matches_reference():
    K, sk = _mods()
    x = torch.randn(5, 1024, generator=torch.Generator().manual_seed(3)) * 2
    w = torch.rand(1024) + 0.5
    xq, xd, xbs = sk.quant256(x.cuda(), w.cuda(), 1e-5)
    assert torch.equal(xbs.cpu().int(), xq.cpu().int().view(5, -1, 32).sum(-1))
    ref = _quant256_ref(R.rmsnorm(x, w, 1e-5))
    got = (xq.cpu().float().view(5, -1, 256) * xd.cpu()[..., None]).view(5, 1024)
    assert torch.allclose(got, ref, atol=2e-2 * ref.abs().max().item() / 127 + 1e-6)
    # a single row comes in the word order of the one-token kernel
    xq1, xd1, xbs1 = sk.quant256(x[:1].cuda(), w.cuda(), 1e-5)
    assert torch.equal(sk.natural_order(xq1).cpu(), xq[:1].cpu()) and torch.equal(xbs1.cpu(), xbs[:1].cpu())


@pytest.mark.parametrize("t", [GGMLType.Q4_K, GGMLType.Q6_K])
@pytest.mark.parametrize("nb", [1, 3, 8, 13, 32])
@pytest.mark.parametrize("ctas", [0, 1, 5])
def test_gemv_sk_matches_reference(t, nb, ctas):
    K, sk = _mods()
    n, k = 208, 1024
    qw = _qw(t, n, k, 11)
    bias = torch.randn(n, generator=torch.Generator().manual_seed(2)) * 0.1
    w = sk.repack(qw, "cuda", bias=bias)
    x = torch.randn(nb, k, generator=torch.Generator().manual_seed(1))
    ref = _quant256_ref(x) @ qw.dequant().t() + bias
    y = sk.gemv([w], x.cuda(), max_ctas=ctas).cpu()          # fp32 rows, quantised inside the kernel
    assert _close(y, ref), (y - ref).abs().max()
    y2 = sk.gemv([w], sk.quant256(x.cuda()), max_ctas=ctas).cpu()      # pre-quantised input
    assert _close(y2, ref), (y2 - ref).abs().max()
    full = x @ qw.dequant().t() + bias
    assert ((y - full).norm() / full.norm()).item() < 2e-2
    out = torch.ones(nb, n, device="cuda")
    sk.gemv([w], x.cuda(), out=out, mode=sk.MODE_ACCUM, max_ctas=ctas)
    assert _close(out.cpu(), ref + 1.0)
    sk.workspace("cuda").check()


@pytest.mark.parametrize("nb", [1, 4])
def test_gemv_sk_norm_prologue_and_segments(nb):
    K, sk = _mods()
    k = 512
    qs = [_qw(GGMLType.Q4_K, 96, k, 1), _qw(GGMLType.Q6_K, 48, k, 2), _qw(GGMLType.Q4_K, 4096, k, 3)]
    ws = [sk.repack(q, "cuda") for q in qs]
    x = torch.randn(nb, k, generator=torch.Generator().manual_seed(5)) * 3
    nw = torch.rand(k, generator=torch.Generator().manual_seed(6)) + 0.5
    xr = _quant256_ref(R.rmsnorm(x, nw, 1e-5))
    ref = torch.cat([xr @ q.dequant().t() for q in qs], 1)
    for ctas in (0, 7, 148):
        for _ in range(2):      # back-to-back launches reuse the hand-over flags
            y = sk.gemv(ws, x.cuda(), norm_w=nw.cuda(), eps=1e-5, max_ctas=ctas).cpu()
            assert y.shape == (nb, 96 + 48 + 4096)
            assert _close(y, ref), (ctas, (y - ref).abs().max())
    sk.workspace("cuda").check()


@pytest.mark.parametrize("act", ["silu", "gelu_tanh", "swiglu_oai"])
def test_gemv_sk_glu(act):
    K, sk = _mods()
    n, k, nb = 256, 512, 3
    qg, qu = _qw(GGMLType.Q4_K, n, k, 1), _qw(GGMLType.Q4_K, n, k, 2)
    g = torch.Generator().manual_seed(9)
    bg, bu = torch.randn(n, generator=g) * 0.1, torch.randn(n, generator=g) * 0.1
    gu = sk.repack(sk.interleave(qg, qu), "cuda", bias=torch.stack([bg, bu], 1).reshape(-1))
    x = torch.randn(nb, k, generator=g) * 3
    xr = _quant256_ref(x)
    ref = R.glu(xr @ qg.dequant().t() + bg, xr @ qu.dequant().t() + bu, act)
    h = sk.gemv([gu], x.cuda(), mode=sk.MODE_GLU, act=act).cpu()
    assert h.shape == (nb, n)
    assert _close(h, ref, 3e-3), (h - ref).abs().max()


def test_gemv_sk_model_shapes():
    """Llama-8B gate/up and down shapes: every SM streams a slice, tiles are split between CTAs."""
    K, sk = _mods()
    dev = "cuda"
    for (n, k, t) in ((2 * 14336, 4096, GGMLType.Q4_K), (4096, 14336, GGMLType.Q6_K)):
        w = torch.randn(512, k, device=dev, generator=torch.Generator(device=dev).manual_seed(n)) * 0.02
        q = QWeight.from_float("w", w, t)
        raw = q.raw.view(512, -1).repeat(n // 512, 1).reshape(-1)
        qw = QWeight("w", t, (n, k), raw)
        u = sk.repack(qw, dev)
        for nb in (1, 8):
            x = torch.randn(nb, k, device=dev)
            ref = _quant256_ref(x) @ q.dequant().t().to(dev)
            ref = ref.repeat(1, n // 512)
            y = sk.gemv([u], x if sk.fits_fused_input(nb, k) else sk.quant256(x))
            assert _close(y.cpu(), ref.cpu()), (n, k, nb, (y - ref).abs().max())
    sk.workspace(dev).check()


@pytest.mark.parametrize("nb", [1, 3])
def test_gemv_chain_runs_dependent_products_in_one_launch(nb):
    """attention-output projection -> gated FFN -> down projection -> next Q/K/V, each phase reading the previous one's output."""
    K, sk = _mods()
    d, f = 512, 1024
    g = torch.Generator().manual_seed(4)
    qo, qg, qu, qd, qq = (_qw(GGMLType.Q4_K, d, d, 1), _qw(GGMLType.Q4_K, f, d, 2), _qw(GGMLType.Q4_K, f, d, 3), _qw(GGMLType.Q6_K, d, f, 4),
                          _qw(GGMLType.Q4_K, 3 * d, d, 5))
    wo, wgu, wd, wq = sk.repack(qo, "cuda"), sk.repack(sk.interleave(qg, qu), "cuda"), sk.repack(qd, "cuda"), sk.repack(qq, "cuda")
    ao = torch.randn(nb, d, generator=g)
    x0 = torch.randn(nb, d, generator=g)
    n1, n2 = torch.rand(d, generator=g) + 0.5, torch.rand(d, generator=g) + 0.5
    # reference
    x1 = x0 + _quant256_ref(ao) @ qo.dequant().t()
    hn = _quant256_ref(R.rmsnorm(x1, n1, 1e-5))
    h = R.glu(hn @ qg.dequant().t(), hn @ qu.dequant().t(), "silu")
    x2 = x1 + _quant256_ref(h) @ qd.dequant().t()
    qkv = _quant256_ref(R.rmsnorm(x2, n2, 1e-5)) @ qq.dequant().t()
    ao_d, n1_d, n2_d = ao.cuda(), n1.cuda(), n2.cuda()      # phases hold raw pointers: the tensors must outlive the launch
    for _ in range(2):      # twice: the barrier counters must be back at zero
        x = x0.cuda().clone()
        hbuf = torch.zeros(nb, f, device="cuda")
        out = torch.zeros(nb, 3 * d, device="cuda")
        ph = [sk.phase([wo], ao_d, x, mode=sk.MODE_ACCUM),
              sk.phase([wgu], x, hbuf, norm_w=n1_d, eps=1e-5, mode=sk.MODE_GLU),
              sk.phase([wd], hbuf, x, mode=sk.MODE_ACCUM),
              sk.phase([wq], x, out, norm_w=n2_d, eps=1e-5)]
        sk.gemv_chain(ph, "cuda")
        sk.workspace("cuda").check()
        assert _close(x.cpu(), x2, 5e-3), (x.cpu() - x2).abs().max()
        assert _close(out.cpu(), qkv, 1e-2), (out.cpu() - qkv).abs().max()


def test_engine_decodes_up_to_32_sequences_in_one_step(tmp_path):
    """A model whose matrices all have a unit layout takes 32 sequences per step; a batched step gives every sequence the
    logits it gets when it is decoded alone, and both agree with the fp32 reference graph."""
    from ollama_b200.engine.b200 import B200Backend, MAX_STREAM_BATCH
    from ollama_b200.engine.backend import TorchBackend, open_model
    from ollama_b200.models.synth import write_synthetic_gguf
    p = str(tmp_path / "m.gguf")
    write_synthetic_gguf(p, "tiny-qwen3", "Q4_K_M")
    g = open_model(p)
    eng = B200Backend(g, "cuda")
    assert eng.max_batch == MAX_STREAM_BATCH and all(L.sk is not None for L in eng.layers) and eng.sk_head is not None
    ref = TorchBackend(g, "cpu")
    n = 32
    eng.alloc(n, 64)
    ref.alloc(n, 64)
    gen = torch.Generator().manual_seed(5)
    prompts = [torch.randint(259, 4096, (5 + s % 7,), generator=gen).tolist() for s in range(n)]
    toks = []
    for s, pr in enumerate(prompts):
        lr = ref.prefill(s, pr, 0)
        eng.prefill(s, pr, 0)
        toks.append(int(lr.argmax()))
    pos = [len(pr) for pr in prompts]
    want = ref.decode(list(range(n)), toks, pos)
    tol = 0.05 * want.abs().max().item()
    for nb in (32, 13, 3, 1):
        got = eng.decode(list(range(nb)), toks[:nb], pos[:nb]).cpu()
        assert (got - want[:nb]).abs().max().item() < tol, nb
        assert eng.decode_argmax(list(range(nb)), toks[:nb], pos[:nb]) == got.argmax(-1).tolist()
    eng.check_waits()


def test_waits_that_ran_out_are_reported_and_cleared(tmp_path):
    """What a launch leaves behind that gave up waiting (set from the host: a status word, a flag set too late) ends the next call that reads results, in steps and prompt passes; the
    calls after it give what they gave before."""
    from ollama_b200.engine.b200 import B200Backend
    from ollama_b200.engine.backend import open_model
    from ollama_b200.models.synth import write_synthetic_gguf
    K, sk = _mods()
    p = str(tmp_path / "m.gguf")
    write_synthetic_gguf(p, "tiny-qwen3", "Q4_K_M")
    eng = B200Backend(open_model(p), "cuda", keep_bf16=True)
    eng.alloc(1, 64)
    assert eng._pass.units and len({id(w) for w in (eng._ws, eng._pass.ws, sk.workspace("cuda"))}) == 3
    prompt = [300, 301, 302, 303, 304]
    want = eng.prefill(0, prompt, 0).clone()
    tok = eng.decode_argmax([0], [5], [5])
    for ws in (eng._ws, eng._pass.ws):
        ws.status[0] = 1
        ws.flags[:] = 1
        with pytest.raises(K.CudaKernelError):
            eng.decode_argmax([0], [5], [5])
        assert int(ws.flags.max()) == 0 and int(ws.status[0]) == 0
        assert torch.equal(eng.prefill(0, prompt, 0), want) and eng.decode_argmax([0], [5], [5]) == tok
        eng.check_waits()
    eng.close()


@pytest.mark.parametrize("segs,k", [([(16, GGMLType.Q4_K)], 256), ([(272, GGMLType.Q6_K), (16, GGMLType.Q4_K), (32, GGMLType.Q6_K)], 512), ([(4096, GGMLType.Q4_K)], 2816)])
@pytest.mark.parametrize("nb", [1, 8, 9, 24, 32])
def test_gemm16_matches_reference(segs, k, nb):
    """Rows in 16-bit activations (kernels/gemm_sk.cu): groups of one tile, groups that matrices of both encodings share, groups split between CTAs; stored, added, normalised, in
    bf16 rows.  Bound: activations keep 2^-12 of a 256-block's largest value (about 3.5 of their deviations), Q6_K codes times scales 2^-12, so 2^-9 of a result's deviation at worst."""
    _, sk = _mods()
    gen = torch.Generator().manual_seed(nb + k)
    ws = [sk.repack(QWeight.from_float("w", torch.randn(n, k, generator=gen) * 0.05, t), "cuda", bias=torch.randn(n, generator=gen)) for n, t in segs]
    W = torch.cat([sk.unit_weights(w) for w in ws]).double()
    bias = torch.cat([w.bias for w in ws]).double()
    W, bias = W.cuda(), bias.cuda()
    x, nw = torch.randn(nb, k, generator=gen).cuda() * 3, torch.rand(k, generator=gen).cuda() + 0.5
    x[0] *= 1e4                                        # rows have scales of their own
    x[-1, :256] = 0

    def check(got, rows):
        ref = rows.double() @ W.t()
        tol = 2 ** -9 * ref.std(1, keepdim=True) + 1e-6
        assert ((got.double() - ref - bias).abs() <= tol + 1e-6 * ref.abs()).all(), ((got.double() - ref - bias).abs() / tol).max()

    check(sk.gemm16(ws, sk.rows16(x), nb), x)
    out = torch.randn(nb, W.shape[0], generator=gen).cuda()
    was = out.clone()
    sk.gemm16(ws, sk.rows16(x), nb, out=out, mode=sk.MODE_ACCUM)
    assert torch.allclose(out - was, sk.gemm16(ws, sk.rows16(x), nb), rtol=1e-4, atol=1e-4 * float(out.abs().max()))
    normed = (x.double() * torch.rsqrt((x.double() ** 2).mean(1, keepdim=True) + 1e-5) * nw.double())
    check(sk.gemm16(ws, sk.rows16(x, nw, 1e-5), nb), normed)
    b16 = x.to(torch.bfloat16)
    check(sk.gemm16(ws, sk.rows16(b16), nb), b16)
    sk.workspace("cuda").check()


@pytest.mark.parametrize("k", [256, 2048, 2304, 4096, 4352])
@pytest.mark.parametrize("t", [GGMLType.Q4_K, GGMLType.Q6_K])
def test_one_row_quantised_inside(k, t):
    """One row that the launch quantises itself, up to 16 blocks (a warp's two in registers) and beyond: the same bits as the row quantised before; normalised, against the statement
    in fp32, from which the few values that lie between two codes may differ by one (1 / 127 of a block's largest, in a row of thousands less than 2e-3 of the result's norm)."""
    _, sk = _mods()
    gen = torch.Generator().manual_seed(k)
    ws = [sk.repack(_qw(t, n, k, n), "cuda") for n in (48, 4096)]
    x, nw = torch.randn(1, k, generator=gen).cuda(), (torch.rand(k, generator=gen) + 0.5).cuda()
    x[0, :min(k - 1, 300)] = 0                         # a block of zeros
    assert torch.equal(sk.gemv(ws, x), sk.gemv(ws, sk.quant256(x)))
    W = torch.cat([sk.unit_weights(w) for w in ws])
    ref = _quant256_ref(R.rmsnorm(x.cpu(), nw.cpu(), 1e-5)).cuda() @ W.t()
    got = sk.gemv(ws, x, norm_w=nw, eps=1e-5)
    assert (got - ref).norm() <= 2e-3 * ref.norm()
    sk.workspace("cuda").check()


@pytest.mark.parametrize("segs,k", [([(16, GGMLType.Q6_K)], 256), ([(2064, GGMLType.Q4_K)], 256), ([(400, GGMLType.Q6_K), (2000, GGMLType.Q4_K)], 1280),
                                    ([(272, GGMLType.Q4_K)], 14336), ([(4096, GGMLType.Q6_K)], 1024), ([(20480, GGMLType.Q4_K)], 768)])
@pytest.mark.parametrize("nb", [2, 16, 17, 33, 48, 49, 64])
def test_gemm16_items_and_rows(segs, k, nb):
    """Every number of 16-row groups of x, with a block a group of matrix rows, groups that end inside a share (finished while the next is under way), shares that end inside a group
    (handed over by either set of warps), one group over all CTAs, and partly filled groups; bound as above."""
    _, sk = _mods()
    gen = torch.Generator().manual_seed(nb + k)
    ws = [sk.repack(QWeight.from_float("w", torch.randn(n, k, generator=gen) * 0.05, t), "cuda") for n, t in segs]
    W = torch.cat([sk.unit_weights(w) for w in ws]).double().cuda()
    x = torch.randn(nb, k, generator=gen).cuda()
    ref = x.double() @ W.t()
    tol = 2 ** -9 * ref.std(1, keepdim=True) + 1e-6
    chunks = sk.rows16(x)
    out = torch.ones(nb, W.shape[0], device="cuda")
    for ctas in (0, 7):                                 # as many CTAs as SMs, and a few with long shares
        assert ((sk.gemm16(ws, chunks, nb, max_ctas=ctas).double() - ref).abs() <= tol).all()
        assert torch.equal(sk.gemm16(ws, chunks, nb, max_ctas=ctas), sk.gemm16(ws, chunks, nb, max_ctas=ctas))
    sk.gemm16(ws, chunks, nb, out=out, mode=sk.MODE_ACCUM)
    assert ((out.double() - 1 - ref).abs() <= tol + 2e-6).all()
    if all(n % 2 == 0 for n, _ in segs):
        glu = torch.nn.functional.silu(ref[:, 0::2]) * ref[:, 1::2]
        assert (sk.gemm16(ws, chunks, nb, mode=sk.MODE_GLU).double() - glu).norm() < 2 ** -9 * glu.norm()
    sk.workspace("cuda").check()


@pytest.mark.parametrize("n,k,nb", [(272, 14336, 3), (1040, 2048, 5), (4096, 4096, 64), (20480, 1024, 17)])
def test_gemm16_parts_are_handed_over_once(n, k, nb):
    """Groups in more parts than finish them, in a few, and with parts of CTAs that go on; outputs of any alignment and stride; a row that is not a number arrives like any other.
    Whatever a launch handed over is taken: the workspace is empty again."""
    _, sk = _mods()
    gen = torch.Generator().manual_seed(n)
    w = sk.repack(QWeight.from_float("w", torch.randn(n, k, generator=gen) * 0.05, GGMLType.Q4_K), "cuda")
    w.bias = torch.randn(n + 1, generator=gen).cuda()[1:]
    x, ws = torch.randn(nb, k, generator=gen).cuda(), sk.workspace("cuda")
    want = sk.gemm16([w], sk.rows16(x), nb)
    ref = x.double() @ sk.unit_weights(w).double().cuda().t() + w.bias.double()
    assert ((want.double() - ref).abs() <= 2 ** -9 * ref.std(1, keepdim=True) + 1e-6).all()
    odd = torch.zeros(nb, n + 3, device="cuda")
    assert torch.equal(sk.gemm16([w], sk.rows16(x), nb, out=odd[:, 1:n + 1]), want) and (odd[:, 0] == 0).all() and (odd[:, n + 1:] == 0).all()
    odd = odd[:, 1:n + 1]
    sk.gemm16([w], sk.rows16(x), nb, out=odd, mode=sk.MODE_ACCUM)
    assert (odd - 2 * want).abs().max() <= 2 ** -20 * want.abs().max()      # two orders of the same sums
    x[nb // 2] = float("nan")
    got = sk.gemm16([w], sk.rows16(x), nb)
    rest = [b for b in range(nb) if b != nb // 2]
    assert torch.equal(got[rest], want[rest]) and got[nb // 2].isnan().all()
    ws.check()
    assert (ws.ws == -1).all()


@pytest.mark.parametrize("n,k,split", [(16, 16384, 1), (6144, 4096, 0), (4000, 1792, 2), (28672, 512, 0)])
@pytest.mark.parametrize("nb", [1, 7])
def test_gemv_parts_are_handed_over_once(n, k, split, nb):
    """A tile in as many parts as it has blocks, and parts of warps that go on: launches one behind the other give the same and leave the workspace empty."""
    _, sk = _mods()
    gen = torch.Generator().manual_seed(n + nb)
    w = sk.repack(QWeight.from_float("w", torch.randn(n, k, generator=gen) * 0.05, GGMLType.Q4_K), "cuda")
    x, ws = torch.randn(nb, k, generator=gen).cuda(), sk.workspace("cuda")
    xin = x if sk.fits_fused_input(nb, k) else sk.quant256(x)
    want = sk.gemv([w], xin, split=split)
    ref = _quant256_ref(x.cpu()).cuda() @ sk.unit_weights(w).cuda().t()
    assert (want - ref).norm() <= 2e-3 * ref.norm()      # values at a rounding tie may be quantised to the code beside
    assert all(torch.equal(sk.gemv([w], xin, split=split), want) for _ in range(3))
    ws.check()
    assert (ws.ws == -1).all()


@pytest.mark.parametrize("hd,H,Hkv", [(128, 8, 2), (64, 12, 4), (32, 8, 8), (256, 3, 1)])
@pytest.mark.parametrize("nb", [2, 16, 17, 64])
def test_attention_merged_into_chunks(hd, H, Hkv, nb):
    """The merge of the splits that writes the output product's chunks gives the bits of the merge and b2_rows16, rows of zeros included; heads of half, of quarter, of eighth and of
    whole blocks, with the tensor-core and with the scalar kernel before it."""
    K, sk = _mods()
    n_ctx, splits = 256, 4
    gen = torch.Generator().manual_seed(nb + hd)
    kc, vc = (torch.randn(nb, Hkv, n_ctx, hd, generator=gen).half().cuda() for _ in range(2))
    q, sinks = torch.randn(nb, H, hd, generator=gen).cuda(), torch.randn(H, generator=gen).cuda()
    pos, slots = torch.randint(0, n_ctx, (nb,), generator=gen, dtype=torch.int32).cuda(), torch.arange(nb, dtype=torch.int32).cuda()
    acc, ml = torch.empty(nb * H * splits * hd, device="cuda"), torch.empty(nb * H * splits * 2, device="cuda")
    out = torch.empty(nb, H * hd, device="cuda")
    chunks = torch.full((sk.rows16_bytes(nb, H * hd),), 0xAA, device="cuda", dtype=torch.uint8)
    a = K.AttnDecodeArgs(K.ptr(q), K.ptr(kc), K.ptr(vc), K.ptr(pos), K.ptr(slots), H, Hkv, n_ctx, splits, hd ** -0.5, 0.0, 0, K.ptr(acc), K.ptr(ml), None, None)
    c = K.AttnCombineArgs(K.ptr(acc), K.ptr(ml), K.ptr(sinks), H, splits, hd, K.ptr(out), None, None)
    assert K.attn_decode_into(a, None, c, nb, hd, False) == 0
    c.out = None
    assert K.attn_decode_into(a, None, c, nb, hd, True, chunks) == 0
    assert torch.equal(chunks, sk.rows16(out, out=torch.full_like(chunks, 0x55)))
    assert K.attn_decode_into(a, None, c, 65, hd, True, chunks) != 0 and K.attn_decode_into(a, None, c, nb, hd, True, chunks[4:]) != 0


def test_gemm16_glu_matches_reference():
    _, sk = _mods()
    gen = torch.Generator().manual_seed(3)
    w = sk.repack(QWeight.from_float("w", torch.randn(1376, 512, generator=gen) * 0.05, GGMLType.Q4_K), "cuda")
    x = torch.randn(19, 512, generator=gen).cuda()
    y = x.double() @ sk.unit_weights(w).double().t()
    ref = torch.nn.functional.silu(y[:, 0::2]) * y[:, 1::2]
    got = sk.gemm16([w], sk.rows16(x), 19, mode=sk.MODE_GLU)
    assert (got.double() - ref).norm() < 2 ** -9 * ref.norm()


def test_steps_of_models_wider_than_the_normalising_pass():
    """Rows longer than ROWS16_MAX_NORM that are normalised on the way stay in the int8 form at any number of sequences (nine: the first that the 16-bit form takes)."""
    from types import SimpleNamespace

    from ollama_b200.engine.b200 import INT8_ROWS, B200Backend
    _, sk = _mods()
    k, nb = sk.ROWS16_MAX_NORM + 256, INT8_ROWS + 1
    gen = torch.Generator().manual_seed(1)
    q = _qw(GGMLType.Q4_K, 32, k, 2)
    x, nw = torch.randn(nb, k, generator=gen), torch.rand(k, generator=gen) + 0.5
    dev = dict(device="cuda")
    be = SimpleNamespace(cfg=SimpleNamespace(norm_eps=1e-5, act="silu", swiglu_alpha=1.702, swiglu_limit=7.0), pdl=False, _n=0, _ws=None, buf=SimpleNamespace(
        x16=torch.zeros(sk.rows16_bytes(nb, k), dtype=torch.uint8, **dev),
        sk_x=(torch.zeros(nb * k, dtype=torch.int8, **dev), torch.zeros(nb * (k // 256), **dev), torch.zeros(nb * (k // 32), dtype=torch.int16, **dev))))
    be._rows_sk = lambda *a, **kw: B200Backend._rows_sk(be, *a, **kw)
    out = torch.zeros(nb, 32, **dev)
    B200Backend._sk(be, [sk.repack(q, "cuda")], x.cuda(), out, nb, norm_w=nw.cuda())
    ref = _quant256_ref(R.rmsnorm(x, nw, 1e-5)) @ q.dequant().t()
    assert _close(out.cpu(), ref), (out.cpu() - ref).abs().max()

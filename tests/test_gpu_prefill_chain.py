"""The kernels between a prompt's matmuls, the K-split sum and the attention of large batches."""
import ctypes as C

import numpy as np
import pytest
import torch

from jitllm_b200 import Q4_K, Q6_K, Device, _lib, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ffn", [(1, 256), (33, 1792), (9, 14336)])
def test_silu_mul_writes_the_gemm_operand(n, ffn):
    """Bit for bit what the f32 rows become on their way into the GEMM: the same output either way."""
    L = _lib.load()
    rng = synth.rng_for(91 + ffn)
    ntok = max(n, 9)
    w = synth.q4k_matrix(rng, 256, ffn)
    st = torch.cuda.current_stream().cuda_stream
    with Device(0) as d:
        d.Reserve(256, ffn, ntok)
        h = d.Upload(Q4_K, w, 256, ffn)
        rows, inv = C.c_void_p(), C.c_void_p()
        assert L.jl_gemm_operand(d.ctx, h.handle, ntok, C.byref(rows), C.byref(inv)) == 0
        gu = torch.randn(ntok, 2 * ffn, device="cuda") * 3
        if n == 1:
            gu[0] = 0                                     # a row of zeros has scale 1
        f32, ref, got = torch.empty(ntok, ffn, device="cuda"), torch.empty(ntok, 256, device="cuda"), torch.empty(ntok, 256, device="cuda")
        assert L.jl_aux_silu_mul(f32.data_ptr(), None, gu.data_ptr(), ntok, ffn, st) == 0
        d.MatMulDev(ref, h, f32, ntok, st)
        assert L.jl_aux_silu_mul_gemm(rows, inv, gu.data_ptr(), ntok, ffn, st) == 0
        assert L.jl_matmul_dev_prepared(d.ctx, got.data_ptr(), 0, h.handle, ntok, st) == 0
        torch.cuda.synchronize()
        assert d.StatusPoll() and torch.equal(got, ref)
        assert L.jl_aux_silu_mul_gemm(rows, inv, gu.data_ptr(), 1, 255, st) == _lib.EINVAL
        assert L.jl_aux_silu_mul_gemm(rows, inv, gu.data_ptr(), 1, 51200 + 256, st) == _lib.DECLINED


# a width of whole super-blocks (the form the operands share) and one that is not
@pytest.mark.parametrize("ffn", [14336, 1000])
def test_silu_mul_rounds_like_f32(ffn):
    """expf (2 units of the last place at most), 1 + e, the quotient and the product: 2 + 3/2 units of 2^-23 and their mixed terms,
    of every result that is not denormal (one under 2^-126 has fewer bits: a gate of -80 times an up of 1e-6)."""
    L = _lib.load()
    gu = torch.randn(64, 2 * ffn, device="cuda", generator=torch.Generator(device="cuda").manual_seed(ffn)) * 4
    gu[0, :ffn] = torch.linspace(-80, 80, ffn, device="cuda")
    out = torch.empty(64, ffn, device="cuda")
    assert L.jl_aux_silu_mul(out.data_ptr(), None, gu.data_ptr(), 64, ffn, torch.cuda.current_stream().cuda_stream) == 0
    ref = torch.nn.functional.silu(gu[:, :ffn].double()) * gu[:, ffn:].double()
    normal = ref.abs() >= 2.0 ** -126
    assert int((~normal).sum()) <= 4 and float(((out.double() - ref).abs() / ref.abs())[normal].max()) <= 3.6 * 2.0 ** -23


def test_silu_mul_gemm_of_two_widths_from_two_threads():
    """Both widths need more than 48 KB of shared memory; neither thread's setting may fail the other's launch."""
    import threading
    L, bad = _lib.load(), []

    def loop(ffn):
        s = torch.cuda.Stream()
        gu = torch.zeros(1, 2 * ffn, device="cuda")
        rows, inv = torch.empty(2, ffn, device="cuda", dtype=torch.float16), torch.empty(1, device="cuda")
        torch.cuda.synchronize()
        for _ in range(3000):
            if L.jl_aux_silu_mul_gemm(rows.data_ptr(), inv.data_ptr(), gu.data_ptr(), 1, ffn, s.cuda_stream) != _lib.OK:
                bad.append(ffn)
        s.synchronize()

    ts = [threading.Thread(target=loop, args=(ffn,)) for ffn in (51200, 12544)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad


@pytest.mark.parametrize("n,slots,hq,hkv,d,max_len", [(1, 1, 2, 1, 2, 1), (37, 3, 4, 2, 64, 40), (130, 2, 32, 8, 128, 130)])
def test_rope_prefill_is_the_single_position_kernel_per_row(n, slots, hq, hkv, d, max_len):
    L = _lib.load()
    st = torch.cuda.current_stream().cuda_stream
    qkv = torch.randn(n, (hq + 2 * hkv) * d, device="cuda")
    ang = torch.arange(max_len, device="cuda").float()[:, None] * torch.rand(d // 2, device="cuda")
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    bf = dict(device="cuda", dtype=torch.bfloat16)
    q, kc, vc = torch.empty(n, hq, d, **bf), torch.full((slots, hkv, max_len, d), 7.0, **bf), torch.full((slots, hkv, max_len, d), 7.0, **bf)
    assert L.jl_aux_rope_prefill(q.data_ptr(), qkv.data_ptr(), kc.data_ptr(), vc.data_ptr(), cos.data_ptr(), sin.data_ptr(), n, slots, hq, hkv,
                                 d, max_len, st) == 0
    q1, k1, v1 = torch.empty_like(q), torch.full((1, hkv, max_len, d), 7.0, **bf), torch.full((1, hkv, max_len, d), 7.0, **bf)
    for r in range(n):
        pos = torch.tensor([r], device="cuda")
        assert L.jl_aux_rope_kv(q1[r].data_ptr(), qkv[r].data_ptr(), k1.data_ptr(), v1.data_ptr(), pos.data_ptr(), cos.data_ptr(), sin.data_ptr(),
                                1, hq, hkv, d, max_len, st) == 0
    torch.cuda.synchronize()
    assert torch.equal(q, q1) and torch.equal(kc, k1.expand_as(kc)) and torch.equal(vc, v1.expand_as(vc))


@pytest.mark.parametrize("T", [9, 17, 130])
def test_prefill_chain_against_the_plain_stack(T):
    """The same prompt with and without the chain: bf16 q, k, v and cache in both, so a few bf16 roundings apart."""
    from jitllm_b200.decoder import Config, Decoder
    cfg = Config(n_layer=2, hidden=512, n_head=4, n_kv=2, head_dim=128, ffn=1024, vocab=512)
    with Device(0) as dev:
        dec = Decoder(dev, cfg, max_batch=3, max_len=136, max_prefill=136, seed=5)
        toks = torch.randint(0, cfg.vocab, (T,), device="cuda")
        assert dec._prefill_chain(toks) is not None
        dec.prefill(toks)
        got, kc, vc = dec.last_logits.clone(), dec.k_cache.clone(), dec.v_cache.clone()
        dec._prefill_chain = lambda tokens: None
        dec.prefill(toks)
        torch.cuda.synchronize()
        rel = lambda a, b: float((a.double() - b.double()).norm() / b.double().norm())
        # two layers, each a bf16 rounding (2^-9) of q, k, v that the other path's f32 sums may take the other way
        assert rel(got, dec.last_logits) <= 2 * 2.0 ** -9 and rel(kc, dec.k_cache) <= 2.0 ** -9 and rel(vc, dec.v_cache) <= 2.0 ** -9
        assert dec._gemm_operand(dec.layers[0]["qkv"], 8) is None        # eight tokens: the decode kernels


@pytest.mark.parametrize("name,rows,k", [("qkv", 1024, 512), ("o", 512, 512), ("gu", 2048, 512), ("down", 512, 1024), ("head", 512, 512)])
@pytest.mark.parametrize("layer", [0, 1])
def test_a_stack_of_mixed_formats(name, rows, k, layer):
    """One Q6_K matrix in a Q4_K stack, in any layer: a prompt, a batched step and a small batch's step run, and agree with
    the plain stack."""
    from jitllm_b200.decoder import Config, Decoder
    cfg = Config(n_layer=2, hidden=512, n_head=4, n_kv=2, head_dim=128, ffn=1024, vocab=512)
    rel = lambda a, b: float((a.double() - b.double()).norm() / b.double().norm())
    # three bf16 roundings (2^-9 each) of q, k, v and the attention's rows that the other path's f32 sums may take the other way
    bar = 3 * 2.0 ** -9
    with Device(0) as dev:
        dec = Decoder(dev, cfg, max_batch=12, max_len=64, max_prefill=40, seed=5)
        w = dev.Upload(Q6_K, synth.matrix(synth.rng_for(6), Q6_K, rows, k), rows, k)
        if name == "head":
            dec.head = w
        else:
            dec.layers[layer][name] = w
        toks = torch.randint(0, cfg.vocab, (40,), device="cuda")
        dec.prefill(toks)
        got, kc, vc = dec.last_logits.clone(), dec.k_cache.clone(), dec.v_cache.clone()
        chain, dec._prefill_chain = dec._prefill_chain, lambda tokens: None
        dec.prefill(toks)
        assert rel(got, dec.last_logits) <= bar and rel(kc, dec.k_cache) <= bar and rel(vc, dec.v_cache) <= bar
        for B in (12, 4):
            pos = torch.tensor([40], device="cuda")
            dec.decode_step_torch(toks[:B], pos)
            ref = dec.last_logits.clone()
            dec.decode_step(toks[:B], pos)
            torch.cuda.synchronize()
            assert dev.StatusPoll() and rel(dec.last_logits, ref) <= bar


# splits that the K range is cut into where tiles leave SMs idle, element counts that are not a multiple of four, every output type
@pytest.mark.parametrize("nrows,k,ntok", [(257, 2048, 9), (1023, 4096, 31), (4096, 4096, 64), (3, 512, 17)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_split_sum(orc, nrows, k, ntok, out_dtype):
    rng = synth.rng_for(95 + nrows)
    w, x = synth.q4k_matrix(rng, nrows, k), synth.activations(rng, ntok, k)
    st = torch.cuda.current_stream().cuda_stream
    with Device(0) as d:
        d.Reserve(nrows, k, ntok)
        h = d.Upload(Q4_K, w, nrows, k)
        assert d.Select(Q4_K, nrows, k, ntok).split_k > 1
        xd = torch.from_numpy(x).cuda()
        buf = torch.full((ntok * nrows + 1,), float("nan"), device="cuda", dtype=out_dtype)
        outs = [buf[o:o + ntok * nrows].view(ntok, nrows) for o in (0, 1)]     # an aligned address and one that is not
        got = []
        for o in outs:
            d.MatMulDev(o, h, xd, ntok, st)
            got.append(o.clone())
        torch.cuda.synchronize()
        assert d.StatusPoll() and torch.equal(*got)
        ref = orc.matmul_f64_blas(Q4_K, w, x, nrows, k, ntok)
        err = np.linalg.norm(got[0].double().cpu().numpy() - ref) / np.linalg.norm(ref)
        assert err <= 2.0 ** -11 + (2.0 ** -8 if out_dtype == torch.bfloat16 else 2.0 ** -11 if out_dtype == torch.float16 else 0)


def test_wave_split_keeps_to_the_scratch():
    """192 tiles on 148 SMs are split three ways (two full waves' worth in four of a third) when the scratch has room for the
    partial planes, and run unsplit when it was sized for less: the same sums to f32 order."""
    nrows, k, ntok = 4096, 14336, 1500
    rng = synth.rng_for(97)
    w, x = synth.q4k_matrix(rng, nrows, k), torch.randn(ntok, k, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    outs = []
    for big in (True, False):
        with Device(0) as d:
            if big:
                d.Reserve(nrows, k, ntok)
            else:                                                      # room for the operand rows only (4 bytes an activation)
                d.Reserve(256, k, ntok)
            h = d.Upload(Q4_K, w, nrows, k)
            outs.append((d.Select(Q4_K, nrows, k, ntok).split_k, torch.empty(ntok, nrows, device="cuda")))
            d.MatMulDev(outs[-1][1], h, x, ntok, st)
            torch.cuda.synchronize()
            assert d.StatusPoll()
    assert outs[0][0] > 1 and outs[1][0] == 1
    a, b = outs[0][1].double(), outs[1][1].double()
    # the tensor core's f32 accumulator truncates: each of the k / 16 additions of a sum can lose one unit (2^-23) of it
    assert float((a - b).norm() / b.norm()) <= k / 16 * 2.0 ** -23


# chunks per CTA from one (the form without a ring) to eight, a cache far longer than its sequences, a last CTA with part of its chunks, sequences that end in any chunk of it
@pytest.mark.parametrize("n,hq,hkv,pos,max_len", [(64, 32, 8, 2048, 2056), (64, 32, 8, 700, 2056), (64, 8, 8, 513, 1500), (33, 16, 8, 1000, 1001),
                                                   (64, 64, 8, 15, 600), (20, 32, 8, 511, 512), (13, 32, 8, 2048, 2056),
                                                   (14, 32, 8, 2048, 2056), (13, 8, 8, 77, 130), (1, 32, 8, 700, 65536)])
def test_attention_of_large_batches(n, hq, hkv, pos, max_len):
    L = _lib.load()
    d, g = 128, hq // hkv
    gen = torch.Generator(device="cuda").manual_seed(pos + n)
    q = (torch.randn(n, hq, d, device="cuda", generator=gen) * 2).to(torch.bfloat16)
    kc = torch.randn(n, hkv, max_len, d, device="cuda", generator=gen).to(torch.bfloat16)
    vc = torch.randn(n, hkv, max_len, d, device="cuda", generator=gen).to(torch.bfloat16)
    kc[:, :, pos + 1:] = float("nan")
    vc[:, :, pos + 1:] = float("nan")
    scratch = torch.zeros(L.jl_aux_attn_scratch_bytes(n, hq, hkv, max_len), device="cuda", dtype=torch.uint8)
    pos_dev, outs = torch.tensor([pos], device="cuda"), []
    for _ in range(2):
        out = torch.full((n, hq * d), float("nan"), device="cuda")
        assert L.jl_aux_attn_decode(out.data_ptr(), None, q.data_ptr(), kc.data_ptr(), vc.data_ptr(), pos_dev.data_ptr(), scratch.data_ptr(), n, hq,
                                    hkv, d, max_len, torch.cuda.current_stream().cuda_stream) == _lib.OK
        outs.append(out)
    torch.cuda.synchronize()
    assert torch.equal(*outs)
    worst = 0.0
    for i in range(0, n, 8):
        qd, kd, vd = q[i:i + 8].double().view(-1, hkv, g, d), kc[i:i + 8, :, :pos + 1].double(), vc[i:i + 8, :, :pos + 1].double()
        p = (torch.einsum("nkgd,nksd->nkgs", qd, kd) / d ** 0.5).softmax(-1)
        ref = torch.einsum("nkgs,nksd->nkgd", p, vd).reshape(-1, hq * d)
        worst = max(worst, float((outs[0][i:i + 8].double() - ref).abs().max() / ref.abs().max()))
    assert worst <= 1e-4          # the bar of the small batches: 16-bit softmax weights, fast exp

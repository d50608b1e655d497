"""The kernels between a prompt's matmuls, the K-split sum and the attention of large batches."""
import ctypes as C

import numpy as np
import pytest
import torch

from jitllm_b200 import Q4_K, Device, _lib, synth

pytestmark = pytest.mark.gpu


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


# chunks per CTA from one to eight, a last CTA with part of its chunks, sequences that end in any chunk of it
@pytest.mark.parametrize("n,hq,hkv,pos,max_len", [(64, 32, 8, 2048, 2056), (64, 32, 8, 700, 2056), (64, 8, 8, 513, 1500), (33, 16, 8, 1000, 1001),
                                                   (64, 64, 8, 15, 600), (20, 32, 8, 511, 512)])
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

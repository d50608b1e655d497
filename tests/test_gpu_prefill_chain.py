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

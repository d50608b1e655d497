"""Q6_K on the row kernel."""
import numpy as np
import pytest
import torch

from jitllm_b200 import K_SIMT, Q6_K, Device, synth

pytestmark = pytest.mark.gpu


def rel(a, ref):
    return float(np.linalg.norm(a - ref) / np.linalg.norm(ref))


def run(dev, w, nrows, k, x):
    ntok = x.shape[0]
    dev.Reserve(nrows, k, ntok)
    h = dev.Upload(Q6_K, w, nrows, k)
    xd = torch.from_numpy(x).cuda()
    out = torch.full((ntok, nrows), float("nan"), device="cuda")
    dev.MatMulDev(out, h, xd, ntok, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert dev.lib.jl_status_poll(dev.ctx, None) == 0
    h.free()
    return out.cpu().numpy()


@pytest.mark.parametrize("nrows,k,ntok", [(1, 256, 1), (5, 512, 1), (3, 256, 2), (1023, 3328, 1), (4096, 14336, 1), (257, 768, 5), (64, 4352, 8), (70, 512, 30)])
def test_row_kernel_matches_float64(orc, nrows, k, ntok):
    """Units left over (k / 64 not a multiple of 32, above and below 256), rows and tokens not a multiple of the block's."""
    rng = synth.rng_for(0xB700 + nrows + k + ntok)
    w, x = synth.matrix(rng, Q6_K, nrows, k), synth.activations(rng, ntok, k)
    ref = orc.matmul_f64(Q6_K, w, x, nrows, k, ntok)
    with Device(0, pin_kernel=K_SIMT) as dev:
        got = run(dev, w, nrows, k, x)
    # 16 products, four runs per unit, k / 16384 units a thread, five shuffles, eight warps: under 64 roundings deep
    assert rel(got, ref) <= 64 * 2.0 ** -24 / 4

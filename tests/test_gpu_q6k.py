"""Q6_K: the integer GEMM that serves 9 tokens and more, and the row kernel below."""
import numpy as np
import pytest
import torch

from jitllm_b200 import K_SIMT, K_TC5, Q6_K, Device, synth

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


# one super-block and one row, tile edges (128 rows; every tile of 16 to 64 tokens), every number of k slices, odd rows and tokens
@pytest.mark.parametrize("nrows,k,ntok", [(1, 256, 9), (37, 512, 16), (128, 768, 17), (129, 1024, 32), (300, 2048, 33), (256, 1280, 64),
                                          (511, 3584, 65), (4096, 4096, 203), (16384, 512, 64), (1024, 14336, 130)])
def test_batch_kernel_matches_float64(orc, nrows, k, ntok):
    rng = synth.rng_for(0xB600 + nrows + k + ntok)
    w, x = synth.matrix(rng, Q6_K, nrows, k), synth.activations(rng, ntok, k)
    ref = orc.matmul_f64(Q6_K, w, x, nrows, k, ntok)
    with Device(0) as dev:
        dev.Reserve(nrows, k, ntok)
        h = dev.Upload(Q6_K, w, nrows, k)
        assert dev.Select(Q6_K, nrows, k, ntok).kernel == K_TC5
        h.free()
        got = run(dev, w, nrows, k, x)
        assert np.array_equal(got, run(dev, w, nrows, k, x))             # fixed order
    # a super-block's sum is exact; joining and scaling it rounds four times, then one addition per super-block and slice
    assert rel(got, ref) <= (4 + k / 256 / 2) * 2.0 ** -24
    with Device(0, pin_kernel=K_SIMT) as dev:
        simt = rel(run(dev, w, nrows, k, x), ref)
    print(f"{nrows}x{k} {ntok} tokens: batch kernel {rel(got, ref):.2e}, row kernel {simt:.2e}")


def test_batch_kernel_in_a_graph_and_on_two_streams(orc):
    """A captured call has a workspace of its own, which a later reserve leaves alone; plain calls on two streams share the
    context's in order."""
    rng = synth.rng_for(80)
    nrows, k, ntok = 256, 1024, 20
    w, xs = synth.matrix(rng, Q6_K, nrows, k), [torch.from_numpy(synth.activations(rng, ntok, k)).cuda() for _ in range(2)]
    with Device(0) as dev:
        dev.Reserve(nrows, k, ntok)
        h = dev.Upload(Q6_K, w, nrows, k)
        outs = [torch.empty(ntok, nrows, device="cuda") for _ in range(3)]
        ss = [torch.cuda.Stream(), torch.cuda.Stream()]
        torch.cuda.synchronize()
        for _ in range(20):
            for i in range(2):
                dev.MatMulDev(outs[i], h, xs[i], ntok, ss[i].cuda_stream)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=ss[0]):
            dev.MatMulDev(outs[2], h, xs[1], ntok, ss[0].cuda_stream)
        dev.Reserve(4096, 4096, 300)
        other = torch.empty(300, nrows, device="cuda")
        dev.MatMulDev(other, h, torch.randn(300, k, device="cuda"), 300, ss[1].cuda_stream)
        g.replay()
        torch.cuda.synchronize()
        assert dev.StatusPoll() and torch.equal(outs[2], outs[1])
        for o, x in zip(outs, xs):
            ref = orc.matmul_f64(Q6_K, w, x.cpu().numpy(), nrows, k, ntok)
            assert rel(o.cpu().numpy(), ref) <= (4 + k / 256 / 2) * 2.0 ** -24
        h.free()


def test_batches_in_graphs_and_on_streams_side_by_side():
    """Two graphs of one context and plain calls on two more streams, all with inputs of their own and no reserve in between, give
    the bits that each gives alone; so do calls on streams that come and go, and a graph after its context's next reserve."""
    rng = synth.rng_for(81)
    nrows, k, ntok, n = 2048, 4096, 60, 4
    w, xs = synth.matrix(rng, Q6_K, nrows, k), [torch.from_numpy(synth.activations(rng, ntok, k)).cuda() for _ in range(n)]
    with Device(0) as dev:
        dev.Reserve(nrows, k, ntok)
        h = dev.Upload(Q6_K, w, nrows, k)
        ref, outs = [torch.empty(ntok, nrows, device="cuda") for _ in range(n)], [torch.empty(ntok, nrows, device="cuda") for _ in range(n)]
        for x, r in zip(xs, ref):
            dev.MatMulDev(r, h, x, ntok, torch.cuda.current_stream().cuda_stream)
        ss = [torch.cuda.Stream() for _ in range(n)]
        torch.cuda.synchronize()
        graphs = [torch.cuda.CUDAGraph() for _ in range(2)]
        for i, g in enumerate(graphs):
            n0 = dev.Stats().launches
            with torch.cuda.graph(g, stream=ss[i]):
                for _ in range(3):
                    dev.MatMulDev(outs[i], h, xs[i], ntok, ss[i].cuda_stream)
            assert dev.Stats().launches - n0 == 6                       # planes and GEMM, not the row kernel

        def together():
            for _ in range(10):
                for i in range(2):
                    with torch.cuda.stream(ss[i]):
                        graphs[i].replay()
                for i in (2, 3):
                    dev.MatMulDev(outs[i], h, xs[i], ntok, ss[i].cuda_stream)
            torch.cuda.synchronize()
            assert dev.StatusPoll()
            for o, r in zip(outs, ref):
                assert torch.equal(o, r)
                o.zero_()

        together()
        dev.Reserve(nrows, k, 3 * ntok)
        together()
        L = dev.lib
        import ctypes as C
        rt = C.CDLL("libcudart.so.12")
        for i in range(40):                                             # a stream's handle may come back, its work is another's
            s = C.c_void_p()
            assert rt.cudaStreamCreateWithFlags(C.byref(s), 1) == 0
            dev.MatMulDev(outs[i % n], h, xs[i % n], ntok, s.value)
            assert rt.cudaStreamDestroy(s) == 0
        torch.cuda.synchronize()
        for o, r in zip(outs, ref):
            assert torch.equal(o, r)
        h.free()


@pytest.mark.parametrize("first", ["upload", "reserve"])
def test_workspace_for_the_widest_matrix_and_the_tokens_reserved(first):
    """Whichever comes first, and whatever width the reserve names."""
    nrows, k, ntok = 64, 1024, 40
    w = synth.matrix(synth.rng_for(82), Q6_K, nrows, k)
    with Device(0) as dev:
        if first == "reserve":
            dev.Reserve(nrows, 512, ntok)
        h = dev.Upload(Q6_K, w, nrows, k)
        if first == "upload":
            assert dev.Select(Q6_K, nrows, k, ntok).kernel == K_SIMT
            dev.Reserve(nrows, 512, ntok)
        assert dev.Select(Q6_K, nrows, k, ntok).kernel == K_TC5
        h.free()


@pytest.mark.parametrize("dist", ["one_huge", "tiny", "huge", "zeros"])
def test_batch_kernel_input_distributions(orc, dist):
    rng = synth.rng_for(78)
    nrows, k, ntok = 64, 2048, 24
    x = rng.standard_normal((ntok, k))
    if dist == "one_huge":
        x[:, ::32] *= 1000.0
    x *= dict(tiny=1e-9, huge=1e9, zeros=0.0).get(dist, 1.0)
    x = x.astype(np.float32)
    w = synth.matrix(rng, Q6_K, nrows, k)
    with Device(0) as dev:
        got = run(dev, w, nrows, k, x)
    ref = orc.matmul_f64(Q6_K, w, x, nrows, k, ntok)
    assert np.array_equal(got, ref) if dist == "zeros" else rel(got, ref) <= (4 + k / 256 / 2) * 2.0 ** -24


# an element of every super-block F times the others and met by weights of zero; full and small scales; every group form
@pytest.mark.parametrize("scales", [127, 16, 4])
@pytest.mark.parametrize("F,ntok", [(1, 40), (30, 9), (100, 20), (150, 25), (400, 48), (1000, 64), (1e4, 50), (1e6, 70)])
def test_batch_kernel_with_wide_super_blocks(orc, scales, F, ntok):
    """The small elements alone make the sums: no further from float64 than an f32 chain of k FMAs, 2.1e-7 here as a random walk of
    its roundings has it (2^-24 / sqrt 3 a step, the partial sums as large as sqrt(i / k) of the last: sqrt(k / 6) of them, half met)."""
    rng = synth.rng_for(0xB900 + scales + ntok)
    nrows, k = 256, 4096
    w = synth.matrix(rng, Q6_K, nrows, k).copy()
    b = w.reshape(-1, 210)
    b[:, 192:208] = rng.integers(-scales, scales + 1, (b.shape[0], 16)).astype(np.int8).view(np.uint8)
    b[:, 5] &= 0xF0                                                     # element 5: code 32, the weight 0
    b[:, 128 + 5] = (b[:, 128 + 5] & 0xFC) | 2
    x = rng.standard_normal((ntok, k)).astype(np.float32)
    x[:, 5::256] = F
    ref = orc.matmul_f64(Q6_K, w, x, nrows, k, ntok)
    with Device(0) as dev:
        got = run(dev, w, nrows, k, x)
    print(f"scales {scales} F {F:g} {ntok} tokens: {rel(got, ref):.2e}")
    assert rel(got, ref) <= 2.1e-7


@pytest.mark.parametrize("scale", [1e-20, 1e-24, 1e-30, 1e-36])
def test_batch_kernel_of_small_activations(orc, scale):
    """Full precision down to the smallest rows (2^-80 and below are added as the row kernel does)."""
    rng = synth.rng_for(86)
    nrows, k, ntok = 64, 1024, 33
    w, x = synth.matrix(rng, Q6_K, nrows, k), (synth.activations(rng, ntok, k) * np.float32(scale)).astype(np.float32)
    with Device(0) as dev:
        got = run(dev, w, nrows, k, x)
    assert rel(got, orc.matmul_f64(Q6_K, w, x, nrows, k, ntok)) <= 12 * 2.0 ** -24


def test_batch_kernel_not_finite():
    """Infinities and NaN give what the row kernel gives, in their own token only."""
    rng = synth.rng_for(79)
    nrows, k, ntok = 130, 1024, 20
    x = synth.activations(rng, ntok, k)
    x[3, 5], x[7, 700], x[11, 9], x[11, 900] = np.inf, np.nan, -np.inf, 1.0
    w = synth.matrix(rng, Q6_K, nrows, k)
    with Device(0) as dev:
        got = run(dev, w, nrows, k, x)
    with Device(0, pin_kernel=K_SIMT) as dev:
        ref = run(dev, w, nrows, k, x)
    assert np.array_equal(np.isnan(got), np.isnan(ref)) and np.array_equal(np.isinf(got), np.isinf(ref))
    fin = np.isfinite(ref)
    assert np.array_equal(got[np.isinf(ref)], ref[np.isinf(ref)]) and rel(got[fin], ref[fin]) <= 1e-6


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


@pytest.mark.parametrize("ntok", [1, 2, 5, 20])
def test_activations_near_the_top_of_f32(orc, ntok):
    """32 x overflows where the weight times x does not: the row kernel's codes are scaled down, the batch kernel's integers know
    no range. (1024 products one after the other at most.)"""
    rng = synth.rng_for(84 + ntok)
    nrows, k = 70, 1024
    w = synth.matrix(rng, Q6_K, nrows, k)
    w.reshape(-1, 210)[:, 208:] = np.array([1e-5], np.float16).view(np.uint8)
    x = (synth.activations(rng, ntok, k).clip(-3, 3) * np.float32(3e37)).astype(np.float32)
    ref = orc.matmul_f64(Q6_K, w, x, nrows, k, ntok)
    assert np.abs(ref).max() < 1e38 and np.abs(x).max() > np.finfo(np.float32).max / 32
    with Device(0) as dev:
        got = run(dev, w, nrows, k, x)
    assert np.isfinite(got).all() and rel(got, ref) <= 1024 * 2.0 ** -24 / 4

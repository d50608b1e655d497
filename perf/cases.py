"""The work a user of this library has it do, as a list of timed cases over its public entry points.

Kinds of case (the "kind" of each dict):

  host     Device.MatVec: one token, host arrays in and out, the weight resident under its host address -- the seam a
           host engine with its own graph binds (one call per matrix and token).
  matmul   Device.MatVecDev (one token) and Device.MatMulDev (several): device tensors in and out. One token is a decode
           step's projection; a few tokens a speculative or small batch; dozens a batched decode; hundreds a prompt.
  moe      Device.MoeDev: router outputs and hidden rows in, the mixture layer added into the residual rows.
  decode   one token for each of `batch` sequences through a stack of Llama-8B-wide blocks and the head: the whole-step
           kernel for one sequence, the per-matmul chain for several.
  prefill  a prompt through the same stack.

Weights are random blocks in the ggml formats, uploaded in `prepare` as a loaded model's would be; a pass is one public call
(for decode and prefill: one step of the decoder). Stacks have 2 to 4 blocks instead of 32, so that they are made quickly:
a pass's time grows linearly with the blocks.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import torch

from jitllm_b200 import ACT_SILU, ACT_SWIGLU_OAI, MXFP4, Q4_0, Q4_K, Q5_0, Q5_1, Q5_K, Q6_K, Q8_0, Device, row_bytes
from jitllm_b200._lib import MOE_ARM_BLOCK_SCALED_X3, MOE_ARM_EXACT, MoeDesc
from jitllm_b200.decoder import Config, Decoder

TYPES = {"q4_k": Q4_K, "q8_0": Q8_0, "mxfp4": MXFP4, "q6_k": Q6_K, "q5_k": Q5_K, "q4_0": Q4_0, "q5_0": Q5_0, "q5_1": Q5_1}
BLOCK_ELEMS = {"q4_k": 256, "q5_k": 256, "q6_k": 256}          # the other formats: 32
DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}

HEAD_DIM, WIDTH, KV_HEADS, FFN, VOCAB = 128, 4096, 8, 14336, 32000


def listed():
    return [
        # the smallest call: a k or v projection at one token, where launch and host latency are most of the time
        dict(name="kv_proj_q4k_1", kind="matmul", type="q4_k", rows=1024, k=4096, tok=1, x="f32", out="f32"),
        # the host-pointer seam at the hidden size
        dict(name="host_q4k_4096", kind="host", type="q4_k", rows=4096, k=4096),
        # mixed files keep half of their down and v matrices (and the head) in Q6_K: decode ...
        dict(name="down_q6k_1", kind="matmul", type="q6_k", rows=4096, k=14336, tok=1, x="f32", out="f32"),
        # ... and the prompt's pass over the same matrix
        dict(name="down_q6k_203", kind="matmul", type="q6_k", rows=4096, k=14336, tok=203, x="f32", out="f32"),
        # a few tokens at a time: speculative decoding, a handful of sequences
        dict(name="ffn_q4k_5", kind="matmul", type="q4_k", rows=14336, k=4096, tok=5, x="f32", out="f32"),
        # batched decode on Q8_0
        dict(name="proj_q8_32", kind="matmul", type="q8_0", rows=4096, k=4096, tok=32, x="f32", out="f32"),
        # a 512-token prompt chunk, bf16 in and out
        dict(name="ffn_q4k_512_bf16", kind="matmul", type="q4_k", rows=14336, k=4096, tok=512, x="bf16", out="bf16"),
        # the mixture layer of a 32-expert model with its own activation and biases: a decode step and a 256-token batch
        dict(name="moe_1", kind="moe", tok=1, experts=32, top_k=4, hidden=2880, ffn=2880, act="oai", arm="exact", h="bf16"),
        dict(name="moe_256", kind="moe", tok=256, experts=32, top_k=4, hidden=2880, ffn=2880, act="oai", arm="exact", h="bf16"),
        # decode at a context of 2048: one sequence and 64
        dict(name="decode_b1", kind="decode", layers=4, batch=1, context=2048),
        dict(name="decode_b64", kind="decode", layers=4, batch=64, context=2048),
        # a long ragged prompt: the largest
        dict(name="prefill_1531", kind="prefill", layers=4, tok=1531),
    ]


def _log(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def _multiple(rng, lo, hi, of):
    return max(of, int(_log(rng, lo, hi) / of + 0.5) * of)


def draw(rng):
    kind = rng.choices(["matmul", "host", "moe", "decode", "prefill"], [6, 1, 2, 1.5, 1])[0]
    if kind in ("matmul", "host"):
        tok = 1 if kind == "host" else rng.choice([1, 1, 1, 2, int(_log(rng, 3, 9)), int(_log(rng, 9, 65)), int(_log(rng, 65, 1025))])
        few = ["q4_k", "q4_k", "q4_k", "q8_0", "q8_0", "mxfp4", "q6_k", "q6_k", "q5_k", "q4_0", "q5_0", "q5_1"]
        many = ["q4_k", "q4_k", "q8_0", "q6_k"]
        t = rng.choice(few if tok <= 8 else many)
        if t == "q6_k":
            tok = min(tok, 203)
        step = BLOCK_ELEMS.get(t, 64 if tok <= 8 else 256)
        rows = int(_log(rng, 256, 16384)) if rng.random() < 0.4 else _multiple(rng, 256, 32768, 64)
        k = _multiple(rng, 512, 14336, step)
        while rows * k > 14336 * 4096:
            rows = rows * 2 // 3
        case = dict(kind=kind, type=t, rows=rows, k=k)
        if kind == "matmul":
            wide = t in ("q4_k", "q8_0") and tok > 8 and k % 256 == 0      # 16-bit activations go to the batched kernels
            case.update(tok=tok, x=rng.choice(["f32", "bf16", "bf16", "f16"]) if wide else "f32")
            case["out"] = rng.choice(["f32", case["x"]]) if wide else "f32"
        return case
    if kind == "moe":
        experts = rng.choice([8, 16, 32])
        return dict(kind=kind, tok=int(_log(rng, 1, 257)), experts=experts, top_k=rng.choice([1, 2, 4, 4]),
                    hidden=_multiple(rng, 512, 2880, 64), ffn=_multiple(rng, 512, 2880, 64), act=rng.choice(["oai", "silu"]),
                    arm=rng.choice(["exact", "exact", "x3"]), h=rng.choice(["bf16", "f32"]))
    if kind == "decode":
        batch = rng.choice([1, 1, int(_log(rng, 2, 9)), int(_log(rng, 9, 65))])
        return dict(kind=kind, layers=rng.choice([2, 3, 4]), batch=batch, context=int(_log(rng, 16, 2049)))
    return dict(kind=kind, layers=rng.choice([2, 3]), tok=int(_log(rng, 17, 1532)))


# ------------------------------------------------------------------------------------------------ inputs

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _set_f16(b, at, values):
    b[:, at:at + 2] = values.to(torch.float16).view(torch.uint8).view(-1, 2)


def _blocks(g, name, n_rows, k):
    """Random blocks of a format on the host, as quantising zero-mean weights of about 0.02 gives them: codes over the whole
    range, block scales that vary by a factor of three, and mins (where the format has them) that centre the codes."""
    per = row_bytes(TYPES[name], BLOCK_ELEMS.get(name, 32))
    n = n_rows * row_bytes(TYPES[name], k) // per
    b = torch.randint(0, 256, (n, per), dtype=torch.uint8, device="cuda", generator=g)
    d = 0.5 + torch.rand(n, device="cuda", generator=g)
    if name in ("q4_k", "q5_k"):
        # weight = d sc q - dmin m: with m = sc and dmin = d x the middle code it is d sc (q - middle). sc and m are 6 bits
        # each: sub-blocks 0..3 in bytes 4..7 (sc) and 8..11 (m), with the two high bits of sub-blocks 4..7 above them,
        # whose low four bits share bytes 12..15 (sc low nibble, m high nibble)
        d *= 9e-5 if name == "q4_k" else 4.5e-5
        _set_f16(b, 0, d)
        _set_f16(b, 2, d * (7.5 if name == "q4_k" else 15.5))
        b[:, 8:12] = b[:, 4:8]
        b[:, 12:16] = (b[:, 12:16] & 15) * 17
    elif name == "q6_k":
        _set_f16(b, 208, d * 1.5e-5)                   # d sc (q - 32), sc int8
    elif name == "mxfp4":
        b[:, 0] = torch.randint(118, 123, (n,), dtype=torch.uint8, device="cuda", generator=g)
    else:
        d *= dict(q8_0=2.7e-4, q4_0=4.3e-3, q5_0=2.2e-3, q5_1=2.2e-3)[name]
        _set_f16(b, 0, d)
        if name == "q5_1":
            _set_f16(b, 2, d * -15.5)                  # d q + m
    return b.cpu().numpy().reshape(n_rows, -1)


class _Held:
    """One device with what is resident on it; given back when the state goes."""

    def __init__(self):
        self.dev, self.weights, self.block = Device(torch.cuda.current_device()), [], None

    def upload(self, name, raw, rows, k, experts=1):
        w = self.dev.Upload(TYPES[name], raw, rows, k, experts)
        self.weights.append(w)
        return w

    def __del__(self):
        try:
            torch.cuda.synchronize()
            if self.block is not None:
                self.block.free()
            for w in self.weights:
                w.free()
            self.dev.Close()
        except Exception:
            pass


def _prepare_host(case, g, held):
    w = _blocks(g, case["type"], case["rows"], case["k"])
    x = torch.randn(case["k"], device="cuda", generator=g).cpu().numpy()
    out = np.zeros(case["rows"], np.float32)
    held.dev.MatVec(out, TYPES[case["type"]], w, x, case["rows"], case["k"])       # the first use uploads the weight
    return dict(w=w, x=x, out=out)


def _prepare_matmul(case, g, held):
    rows, k, tok = case["rows"], case["k"], case["tok"]
    held.dev.Reserve(rows, k, tok)
    w = held.upload(case["type"], _blocks(g, case["type"], rows, k), rows, k)
    x = torch.randn(tok, k, device="cuda", generator=g).to(DTYPES[case["x"]])
    return dict(w=w, x=x, out=torch.empty(tok, rows, device="cuda", dtype=DTYPES[case["out"]]))


def _prepare_moe(case, g, held):
    E, H, F, tok = case["experts"], case["hidden"], case["ffn"], case["tok"]
    held.dev.MoeReserve(tok, E, case["top_k"], H, F)
    gate, up, down = (held.upload("mxfp4", _blocks(g, "mxfp4", E * r, k), r, k, E) for r, k in ((F, H), (F, H), (H, F)))
    biases = [torch.randn(E, n, device="cuda", generator=g) * 0.1 if case["act"] == "oai" else None for n in (F, F, H)]
    d = MoeDesc(struct_size=C.sizeof(MoeDesc), type=MXFP4, n_expert=E, top_k=case["top_k"], hidden=H, ffn=F,
                act=ACT_SWIGLU_OAI if case["act"] == "oai" else ACT_SILU, norm=1, scale=1.0, gate=gate.handle, up=up.handle,
                down=down.handle, arm=MOE_ARM_BLOCK_SCALED_X3 if case["arm"] == "x3" else MOE_ARM_EXACT)
    for field, b in zip(("gate_bias", "up_bias", "down_bias"), biases):
        if b is not None:
            setattr(d, field, b.data_ptr())
    return dict(desc=d, biases=biases, h=torch.randn(tok, H, device="cuda", generator=g).to(DTYPES[case["h"]]),
                logits=torch.randn(tok, E, device="cuda", generator=g), residual=torch.randn(tok, H, device="cuda", generator=g),
                out=torch.empty(tok, H, device="cuda"), sel=torch.empty(tok, case["top_k"], dtype=torch.int32, device="cuda"),
                wt=torch.empty(tok, case["top_k"], device="cuda"))


def _decoder(case, seed, g, held, batch, positions):
    cfg = Config(n_layer=0, hidden=WIDTH, n_head=WIDTH // HEAD_DIM, n_kv=KV_HEADS, head_dim=HEAD_DIM, ffn=FFN, vocab=VOCAB)
    dec = Decoder(held.dev, cfg, batch, positions, seed=seed, max_prefill=case.get("tok", 1))
    dec.head.free()
    # a loaded model in place of the harness's own random weights (made on the host, and not centred)
    shapes = dict(qkv=(WIDTH + 2 * KV_HEADS * HEAD_DIM, WIDTH), o=(WIDTH, WIDTH), gu=(2 * FFN, WIDTH), down=(WIDTH, FFN))
    dec.layers = [{name: held.upload("q4_k", _blocks(g, "q4_k", r, k), r, k) for name, (r, k) in shapes.items()}
                  for _ in range(case["layers"])]
    dec.head = held.upload("q4_k", _blocks(g, "q4_k", VOCAB, WIDTH), VOCAB, WIDTH)
    dec.norm_w.copy_(torch.rand(WIDTH, device="cuda", generator=g) + 0.5)
    cfg.n_layer = case["layers"]
    dec.k_cache = torch.zeros(cfg.n_layer, batch, KV_HEADS, positions, HEAD_DIM, device="cuda", dtype=torch.bfloat16)
    dec.v_cache = torch.zeros_like(dec.k_cache)
    return dec


def _prepare_decode(case, seed, g, held):
    B, ctx = case["batch"], case["context"]
    dec = _decoder(case, seed, g, held, B, ctx + 8)
    dec.k_cache.normal_(generator=g)
    dec.v_cache.normal_(generator=g)
    if B == 1:
        if not dec.prep_block_kernel():
            raise RuntimeError("the whole-step kernel declined the stack")
        held.block = dec.block
    return dict(dec=dec, tok=torch.randint(0, VOCAB, (B,), device="cuda", generator=g),
                pos=torch.full((1,), ctx, dtype=torch.int64, device="cuda"))


def _prepare_prefill(case, seed, g, held):
    dec = _decoder(case, seed, g, held, 1, (case["tok"] + 63) // 64 * 64)
    return dict(dec=dec, prompt=torch.randint(0, VOCAB, (case["tok"],), device="cuda", generator=g))


def prepare(case, seed):
    held, g = _Held(), _gen(seed)
    if case["kind"] in ("decode", "prefill"):
        make = _prepare_decode if case["kind"] == "decode" else _prepare_prefill
        state = make(case, seed, g, held)
    else:
        state = dict(host=_prepare_host, matmul=_prepare_matmul, moe=_prepare_moe)[case["kind"]](case, g, held)
    state.update(case=case, held=held)
    return state


# -------------------------------------------------------------------------------------------------- pass

def run(s):
    case, dev = s["case"], s["held"].dev
    kind = case["kind"]
    if kind == "host":
        if not dev.MatVec(s["out"], TYPES[case["type"]], s["w"], s["x"], case["rows"], case["k"]):
            raise RuntimeError(dev.Err())
        return s["out"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "matmul":
        if case["tok"] == 1:
            dev.MatVecDev(s["out"], s["w"], s["x"], 1, stream)
        else:
            dev.MatMulDev(s["out"], s["w"], s["x"], case["tok"], stream)
        return s["out"]
    if kind == "moe":
        s["out"].copy_(s["residual"])                  # the layer adds into the residual rows
        dev.MoeDev(s["out"], s["h"], s["logits"], case["tok"], s["desc"], s["sel"], s["wt"], stream)
        return dict(out=s["out"], sel=s["sel"], wt=s["wt"])
    dec = s["dec"]
    if kind == "decode":
        tok = dec.decode_step_block(s["tok"], s["pos"]) if case["batch"] == 1 else dec.decode_step(s["tok"], s["pos"])
    else:
        tok = dec.prefill(s["prompt"])
    # the chosen token's own logit stands for its id: two nearly equal logits may swap places
    return dict(chosen=dec.last_logits.gather(1, tok.view(-1, 1)), logits=dec.last_logits, k=dec.k_cache, v=dec.v_cache)


# ------------------------------------------------------------------------------------- work and tolerance

def work(case):
    kind = case["kind"]
    size = dict(f32=4, bf16=2, f16=2)
    if kind in ("host", "matmul"):
        tok, rows, k = case.get("tok", 1), case["rows"], case["k"]
        return dict(bytes=rows * row_bytes(TYPES[case["type"]], k) + tok * (k * size[case.get("x", "f32")] + rows * size[case.get("out", "f32")]),
                    flops=2 * tok * rows * k)
    if kind == "moe":
        E, K, H, F, tok = case["experts"], case["top_k"], case["hidden"], case["ffn"], case["tok"]
        hit = E * (1 - (1 - K / E) ** tok)             # experts that at least one token chooses
        return dict(bytes=hit * (2 * F * row_bytes(MXFP4, H) + H * row_bytes(MXFP4, F)) + tok * (H * (size[case["h"]] + 8) + E * 4 + K * 8),
                    flops=6 * tok * K * H * F)
    kv = KV_HEADS * HEAD_DIM
    per_layer = (WIDTH + 2 * kv) * WIDTH + WIDTH * WIDTH + 3 * FFN * WIDTH
    weights, layers = per_layer * case["layers"], case["layers"]
    if kind == "decode":
        B, seen = case["batch"], case["context"] + 1
        return dict(bytes=(weights + VOCAB * WIDTH) * 144 / 256 + layers * B * 2 * kv * 2 * seen + B * (WIDTH * 2 + VOCAB * 4),
                    flops=2 * B * (weights + VOCAB * WIDTH) + layers * B * 4 * WIDTH * seen)
    T = case["tok"]
    return dict(bytes=(weights + VOCAB * WIDTH) * 144 / 256 + layers * T * 2 * kv * 2 + T * WIDTH * 2 + VOCAB * 4,
                flops=2 * (T * weights + VOCAB * WIDTH) + layers * 2 * WIDTH * T * T)


def tolerance(case):
    """About four times the error against float64 sums over the same quantised weights (2-norm)."""
    kind = case["kind"]
    if kind == "decode":      # bf16 q, k, v and cache through the blocks: 4.5e-3 against the same step with PyTorch attention
        return {"rel": 1e-2}
    if kind == "prefill":     # the same, against float64 with q, k and v rounded to bf16: 4.5e-3 to 5.8e-3
        return {"rel": 2e-2}
    if kind == "moe":         # exact weights, f32 sums: 3.8e-6; 12-bit activations: 2.2e-5
        return {"rel": 1e-4 if case["arm"] == "x3" else 1.6e-5}
    if case["type"] not in ("q4_k", "q8_0"):
        return {"rel": 1e-5}  # f32 weights and sums: 1e-7 to 4e-7 by row kernels; sums in another order
    if case.get("out") == "bf16":
        return {"rel": 7e-3}  # the output's rounding: 1.7e-3
    if case.get("tok", 1) <= (8 if case["type"] == "q4_k" else 32) and case.get("x", "f32") == "f32":
        return {"rel": 1.1e-4}                         # 16-bit activations: 2.7e-5
    return {"rel": 1.2e-3 if case.get("out") == "f16" else 8e-4}       # weights rounded once to f16: 2.1e-4 (f16 out 2.9e-4)

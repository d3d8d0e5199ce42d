"""Performance cases of the Q8 decode path, run through the package's public entry points.

A case is a dict of plain values; its "kind" says which call it makes:

  gemv     q8Gemv: one projection of a batch-1 program
  gemm     q8Gemm (bf16 activations and results, any epilogue) or q8GemmF32 (f32 in and out)
  attn     gqaDecodeAttn, or gqaDecodeAttnFused (RoPE and KV append inside)
  decode   a model that decodes: one decodeSteps call, or one decodeStep call per token
  prefill  a model that takes prompts: prefill, or prefillRagged for prompts of different lengths

Weights, caches and activations come from the package's own seeded generator with the
distributions of its benchmark: int8 uniform in [-127, 127], block scales uniform in [1e-3, 1e-2],
activations and KV rows N(0, 1), model weights N(0, 0.02) quantised to Q8 blocks of 32.
"""
import math
import random

import numpy as np
import torch

from logicaffeine_b200 import llm

# The two model shapes of the benchmark.  "32b" is cut to the first `layers` of its 64 layers, so
# that three models fit the card at once; a layer and the head have their full sizes.
MODELS = {
    "0.5b": dict(layers=24, hidden=896, h_q=14, h_kv=2, head_dim=64, ffn=4864, vocab=151936, tied_embeddings=1),
    "32b": dict(layers=64, hidden=5120, h_q=64, h_kv=8, head_dim=128, ffn=27648, vocab=152064, tied_embeddings=0),
}
ACT = {"f32": llm.F32, "f16": llm.F16, "bf16": llm.BF16}


def listed():
    return [
        # The smallest call: one square projection at batch 1, where launch and host time count.
        dict(name="gemv_4096", kind="gemv", n=4096, k=4096),
        # The largest matrix a batch-1 program multiplies: the lm_head of the 32b shape.
        dict(name="gemv_lm_head", kind="gemv", n=152064, k=5120),
        # A 64-token decode batch through a 7B-sized FFN up-projection.
        dict(name="gemm_ffn_up_m64", kind="gemm", m=64, n=18944, k=3584, dtype="bf16", epilogue=0),
        # The down-projection that a rank of eight holds of the same FFN: 18944 / 8 columns is no
        # multiple of 128.  f32 in and out, as between the kernels of a step.
        dict(name="gemm_down_shard_f32", kind="gemm", m=64, n=3584, k=2368, dtype="f32", epilogue=0),
        # A prompt's 2048 tokens through gate and up with the SwiGLU epilogue: the compute-bound end.
        dict(name="gemm_gate_up_prompt", kind="gemm", m=2048, n=37888, k=3584, dtype="bf16", epilogue=2),
        # A decode batch of 32 at 4096 cached positions: rotate, append and attend in one call.
        dict(name="attn_append_b32_4096", kind="attn", b=32, h_q=28, h_kv=4, d=128, ctx=4096, fused=True, ragged=False),
        # A few sequences of very different lengths over a small model's heads.
        dict(name="attn_ragged_b7", kind="attn", b=7, h_q=14, h_kv=2, d=64, ctx=2000, fused=False, ragged=True),
        # The 0.5B shape, batch 16, after its 128-token prompts: many small launches per step.
        dict(name="decode_0.5b_b16", kind="decode", model="0.5b", layers=24, batch=16, ctx=128, steps=16,
             stream=False, temperature=0.0, top_k=0),
        # One conversation, token by token as they are shown, sampled with temperature and top-k.
        dict(name="decode_0.5b_b1_sampled", kind="decode", model="0.5b", layers=24, batch=1, ctx=1000, steps=8,
             stream=True, temperature=0.8, top_k=50),
        # Throughput decode of the 32b shape: batch 64 at context 2048.
        dict(name="decode_32b_b64", kind="decode", model="32b", layers=8, batch=64, ctx=2048, steps=4,
             stream=False, temperature=0.0, top_k=0),
        # Prompts of different lengths in one batch, as they arrive.
        dict(name="prefill_0.5b_ragged", kind="prefill", model="0.5b", layers=24, batch=16, t=128, ragged=True, act="f32"),
        # 4096 prompt tokens of equal-length prompts through the 32b shape.
        dict(name="prefill_32b_b8_512", kind="prefill", model="32b", layers=4, batch=8, t=512, ragged=False, act="f32"),
    ]


def _log_int(rng, lo, hi):
    """An integer of [lo, hi], uniform over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _blocks(rng, lo, hi):
    """A multiple of the Q8 block of [lo, hi], uniform over its logarithm."""
    return 32 * _log_int(rng, lo // 32, hi // 32)


def draw(rng):
    kind = rng.choice(["gemv", "gemm", "gemm", "attn", "attn", "decode", "prefill"])
    while True:
        if kind == "gemv":
            c = dict(kind=kind, n=_log_int(rng, 256, 152064), k=_blocks(rng, 512, 16384))
            if c["n"] * c["k"] <= 152064 * 5120:
                return c
        elif kind == "gemm":
            c = dict(kind=kind, m=_log_int(rng, 1, 4096), n=_log_int(rng, 256, 38000), k=_blocks(rng, 512, 27648),
                     dtype=rng.choice(["bf16", "f32"]), epilogue=0)
            if rng.random() < 0.75:  # widths of models are mostly multiples of 128; what a rank holds often is not
                c["n"], c["k"] = -(-c["n"] // 128) * 128, -(-c["k"] // 128) * 128
            if c["dtype"] == "bf16":
                c["epilogue"] = rng.choice([0, 1, 2])
                c["n"] += c["n"] % 2 if c["epilogue"] == 2 else 0
            if c["m"] * c["n"] * c["k"] <= 2048 * 37888 * 3584:
                return c
        elif kind == "attn":
            h_q, h_kv, d = rng.choice([(28, 4, 128), (64, 8, 128), (16, 2, 128), (8, 1, 128), (14, 2, 64)])
            c = dict(kind=kind, b=_log_int(rng, 1, 64), h_q=h_q, h_kv=h_kv, d=d, ctx=_log_int(rng, 32, 8192),
                     fused=rng.random() < 0.5, ragged=rng.random() < 0.5)
            if c["b"] * h_kv * d * c["ctx"] <= 32 * 4 * 128 * 4096:
                return c
        elif kind == "decode":
            small = rng.random() < 0.7
            stream = rng.random() < 0.4
            sampled = rng.random() < 0.4
            c = dict(kind=kind, model="0.5b" if small else "32b", layers=24 if small else rng.randint(2, 8),
                     batch=_log_int(rng, 1, 64), ctx=_log_int(rng, 16, 2048), steps=rng.randint(1, 16 if small else 4),
                     stream=stream, temperature=0.8 if sampled else 0.0, top_k=rng.choice([0, 50]) if sampled else 0)
            return c
        else:
            small = rng.random() < 0.6
            ragged = rng.random() < 0.4
            c = dict(kind=kind, model="0.5b" if small else "32b", layers=24 if small else rng.randint(1, 4),
                     batch=_log_int(rng, 1, 32), t=_log_int(rng, 16, 128 if ragged else 1024), ragged=ragged,
                     act="f32" if ragged else rng.choice(["f32", "f32", "f16", "bf16"]))
            if c["batch"] * c["t"] <= 4096:
                return c


class _Memory:
    """A device buffer as torch takes it; a tensor over it keeps the buffer alive."""

    def __init__(self, buf, code, shape):
        self.buf = buf
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr=code, data=(buf.ptr(), False), version=3)


def _view(buf, dtype, shape):
    """A torch tensor over a device buffer's memory."""
    code = {torch.float32: "<f4", torch.float16: "<f2", torch.bfloat16: "<i2", torch.int32: "<i4"}[dtype]
    t = torch.as_tensor(_Memory(buf, code, shape), device="cuda:0")
    return t.view(torch.bfloat16) if dtype == torch.bfloat16 else t


def _filled(dtype, kind, seed, stream, count, a=0.0, b=1.0):
    size = {llm.F32: 4, llm.F16: 2, llm.BF16: 2, llm.I8: 1, llm.I32: 4}[dtype]
    buf = llm.DeviceBuffer(count * size)
    llm.synthFill(buf, dtype, kind, seed, stream, 0, count, a, b)
    return buf


def _weights(n, k, seed):
    return _filled(llm.I8, 0, seed, 1, n * k), _filled(llm.F32, 1, seed, 2, n * (k // 32), 1e-3, 1e-2)


def _spread(count, most, seed):
    """Lengths spread evenly over [1, most], in an order that the seed gives."""
    v = [1 + int((most - 1) * (i + 1) / count) for i in range(count)]
    random.Random(seed).shuffle(v)
    return np.array(v, np.int32)


def _model(case, l_max, seed):
    cfg = dict(MODELS[case["model"]], layers=case["layers"], batch=case["batch"], l_max=l_max, seed=seed, init_std=0.02,
               act_dtype=ACT[case.get("act", "f32")])
    return llm.Llm(**cfg)


def _tokens(case, shape, seed):
    return np.random.RandomState(seed & 0x7FFFFFFF).randint(0, MODELS[case["model"]]["vocab"], shape).astype(np.int32)


def prepare(case, seed):
    c = case
    if c["kind"] == "gemv":
        q, s = _weights(c["n"], c["k"], seed)
        x = _filled(llm.F32, 2, seed, 3, c["k"])
        y = llm.DeviceBuffer(c["n"] * 4)
        return dict(case=c, args=(q, s, x, y, c["n"], c["k"]), out=_view(y, torch.float32, (c["n"],)))
    if c["kind"] == "gemm":
        m, n, k = c["m"], c["n"], c["k"]
        q, s = _weights(n, k, seed)
        if c["dtype"] == "f32":
            a, out = _filled(llm.F32, 2, seed, 3, m * k), llm.DeviceBuffer(m * n * 4)
            return dict(case=c, args=(a, q, s, out, m, n, k), out=_view(out, torch.float32, (m, n)))
        n_out = n // 2 if c["epilogue"] == llm.EPI_SWIGLU else n
        a, out = _filled(llm.BF16, 2, seed, 3, m * k), llm.DeviceBuffer(m * n_out * 2)
        aux = _filled(llm.BF16, 2, seed, 4, m * n) if c["epilogue"] == llm.EPI_RESIDUAL else None
        return dict(case=c, args=(a, q, s, out, m, n, k, c["epilogue"], aux), out=_view(out, torch.bfloat16, (m, n_out)))
    if c["kind"] == "attn":
        b, h_q, h_kv, d = c["b"], c["h_q"], c["h_kv"], c["d"]
        l_max = c["ctx"] + 1
        kc, vc = (_filled(llm.F16, 2, seed, j, b * h_kv * l_max * d) for j in (1, 2))
        q = _filled(llm.F16, 2, seed, 3, b * h_q * d)
        lens = _spread(b, c["ctx"], seed) if c["ragged"] else np.full(b, c["ctx"], np.int32)
        seq, o = llm.DeviceBuffer.from_host(lens), llm.DeviceBuffer(b * h_q * d * 2)
        st = dict(case=c, out=_view(o, torch.float16, (b, h_q, d)))
        tail = (b, h_q, h_kv, d, l_max, 1.0 / math.sqrt(d))
        if not c["fused"]:
            return dict(st, args=(q, kc, vc, seq, o) + tail)
        kn, vn = (_filled(llm.F16, 2, seed, j, b * h_kv * d) for j in (4, 5))
        tab = llm.DeviceBuffer.from_host(llm.ropeTable(l_max, d, 1e6))
        cache = [_view(x, torch.float16, (b, h_kv, l_max, d)) for x in (kc, vc)]
        return dict(st, args=(q, kn, vn, kc, vc, tab, seq, o) + tail, cache=cache, seq=_view(seq, torch.int32, (b,)),
                    lens=torch.from_numpy(lens).cuda())
    if c["kind"] == "decode":
        m = _model(c, c["ctx"] + c["steps"] + 1, seed)
        m.synthKv(c["ctx"], seed)
        m.setSampling(c["temperature"], seed, c["top_k"])
        return dict(case=c, model=m, tokens=_tokens(c, (c["batch"],), seed))
    m = _model(c, c["t"] + 16, seed)
    st = dict(case=c, model=m, tokens=_tokens(c, (c["batch"], c["t"]), seed))
    return dict(st, lens=_spread(c["batch"], c["t"], seed)) if c["ragged"] else st


def run(state):
    c = state["case"]
    if c["kind"] == "gemv":
        llm.q8Gemv(*state["args"])
        return state["out"]
    if c["kind"] == "gemm":
        (llm.q8GemmF32 if c["dtype"] == "f32" else llm.q8Gemm)(*state["args"])
        return state["out"]
    if c["kind"] == "attn":
        if not c["fused"]:
            llm.gqaDecodeAttn(*state["args"])
            return state["out"]
        state["seq"].copy_(state["lens"])  # the call advances the lengths: every pass starts at the same ones
        llm.gqaDecodeAttnFused(*state["args"])
        return [state["out"], state["seq"]] + state["cache"]
    m = state["model"]
    if c["kind"] == "decode":
        m.setSeqLen(c["ctx"])
        m.setTokens(state["tokens"])
        if c["stream"]:
            return [m.decodeStep() for _ in range(c["steps"])]
        return m.decodeSteps(c["steps"])
    if c["ragged"]:
        # the prompts' own next tokens stay inside the model: the step after them shows the first ids
        m.prefillRagged(state["tokens"], state["lens"])
        return [m.decodeStep(), m.readSeqLen()]
    m.prefill(state["tokens"])
    return m.readLogits()


def _weight_count(case):
    """Weights of the GEMMs of one step: the layers, and the lm_head."""
    w = MODELS[case["model"]]
    h, nq, nkv, f = w["hidden"], w["h_q"] * w["head_dim"], w["h_kv"] * w["head_dim"], w["ffn"]
    return case["layers"] * ((nq + 2 * nkv) * h + h * nq + 3 * f * h), w["vocab"] * h


def work(case):
    c = case
    if c["kind"] == "gemv":
        return dict(bytes=c["n"] * c["k"] * 1.125 + 4 * (c["n"] + c["k"]), flops=2 * c["n"] * c["k"])
    if c["kind"] == "gemm":
        m, n, k, size = c["m"], c["n"], c["k"], 4 if c["dtype"] == "f32" else 2
        n_out = n // 2 if c["epilogue"] == llm.EPI_SWIGLU else n
        aux = n if c["epilogue"] == llm.EPI_RESIDUAL else 0
        return dict(bytes=n * k * 1.125 + size * m * (k + n_out + aux), flops=2 * m * n * k)
    if c["kind"] == "attn":
        b, h_q, h_kv, d, new = c["b"], c["h_q"], c["h_kv"], c["d"], 1 if c["fused"] else 0
        positions = int(_spread(b, c["ctx"], 0).sum()) if c["ragged"] else b * c["ctx"]
        return dict(bytes=4 * h_kv * d * (positions + 2 * new * b) + 4 * b * h_q * d,
                    flops=4 * h_q * d * (positions + new * b))
    w = MODELS[c["model"]]
    layers, head = _weight_count(c)
    attn_row = 4 * w["h_kv"] * w["head_dim"] * c["layers"]       # bytes of one cached position in all layers
    attn_ops = 4 * w["h_q"] * w["head_dim"] * c["layers"]        # operations of one query on one position
    if c["kind"] == "decode":
        b, steps = c["batch"], c["steps"]
        positions = b * sum(c["ctx"] + i + 1 for i in range(steps))
        return dict(bytes=steps * (layers + head) * 1.125 + attn_row * positions,
                    flops=2 * b * steps * (layers + head) + attn_ops * positions)
    lens = [int(v) for v in _spread(c["batch"], c["t"], 0)] if c["ragged"] else [c["t"]] * c["batch"]
    rows, pairs = sum(lens), sum(n * (n + 1) // 2 for n in lens)
    flops = 2 * rows * layers + 2 * c["batch"] * head + attn_ops * pairs
    nbytes = (layers + head) * 1.125 + 2 * attn_row * rows
    if c["ragged"]:  # and the decode step after the prompts
        flops += 2 * c["batch"] * (layers + head) + attn_ops * (rows + c["batch"])
        nbytes += (layers + head) * 1.125 + attn_row * (rows + c["batch"])
    else:
        nbytes += 4 * c["batch"] * w["vocab"]
    return dict(bytes=nbytes, flops=flops)


def tolerance(case):
    c = case
    if c["kind"] == "gemv":
        return dict(rel=1e-5)                      # f32 sums
    if c["kind"] == "gemm":
        return dict(rel=1e-5) if c["dtype"] == "f32" else dict(rel=4e-3)   # bf16 results: half a last place is 2^-9
    if c["kind"] == "attn":
        return dict(rel=1e-3)                      # fp16 results: half a last place is 2^-11
    if c["kind"] == "decode" or c["ragged"]:
        return dict(rel=0.0, differ=0.01)          # token ids: a near tie of two logits may fall either way
    return dict(rel=1e-3 if c["act"] == "f32" else 2e-2)  # f32 logits over an fp16 KV cache, or 16-bit activations

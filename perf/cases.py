"""What is measured: the work a program has this package do, through its public entry points.

The package is an inference path, so every case is a forward pass: whole encoders (W8A8 and fp16; eager calls, captured
graphs, unpadded batches, host buffers in and out) and the operators of the ``zenith_cuda`` surface and the quantized /
fp16 Linears called on their own.  Weights are random with the distributions of an initialised encoder and its
calibrated scales; token ids are uniform over the vocabulary; key lengths leave a few padding positions per sequence
(or, for unpadded batches, a quarter to all of the positions).

A case is a dict of plain values: ``kind`` and that kind's sizes and options.
"""
from __future__ import annotations

import math

import torch

from zenith_b200 import ops, zenith_cuda
from zenith_b200.encoder import BERT_BASE, BERT_LARGE, Fp16Encoder, Int8Encoder, Int8Scales
from zenith_b200.serve import HostPipeline

DEVICE = "cuda:0"
MODELS = {"base": BERT_BASE, "large": BERT_LARGE}
HOST_BATCHES = 4  # batches per pass of a host-buffer stream, as many as the pipeline holds

# (out features, in features) of the projections of the two encoder configurations
PROJECTIONS = ((2304, 768), (768, 768), (3072, 768), (768, 3072), (3072, 1024), (1024, 1024), (4096, 1024), (1024, 4096))


def _encoder(name, precision, model, batch, seq, form):
    return {"name": name, "kind": "encoder", "precision": precision, "model": model, "batch": batch, "seq": seq, "form": form}


def listed():
    return [
        # an interactive query: one short sentence through the plain call, where launches and latency are everything
        _encoder("int8_base_1x24_forward", "int8", "base", 1, 24, "forward"),
        # a handful of requests gathered by a server into one odd-sized captured batch
        _encoder("int8_base_5x77_replay", "int8", "base", 5, 77, "replay"),
        # the headline configuration fed from and drained to pinned host memory
        _encoder("int8_base_32x128_host", "int8", "base", 32, 128, "host"),
        # offline embedding of documents of mixed length: no work for padding
        _encoder("int8_base_48x256_unpadded", "int8", "base", 48, 256, "unpadded"),
        # one GPU's shard of the large model's batch
        _encoder("int8_large_32x384_replay", "int8", "large", 32, 384, "replay"),
        # the unquantized encoder at the headline shape
        _encoder("fp16_base_32x128_replay", "fp16", "base", 32, 128, "replay"),
        # one quantized Linear + GELU on fp32 activations
        {"name": "linear_int8_128x3072x768", "kind": "linear", "precision": "int8", "m": 128, "n": 3072, "k": 768,
         "act": "gelu", "out": "float32"},
        # the attention sweep: a causal pass at head size 64 and the longest full pass at head size 128
        {"name": "attention_8x16x2048x64_causal", "kind": "attention", "dtype": "float16", "batch": 8, "heads": 16, "seq": 2048,
         "dim": 64, "causal": True, "padded": False},
        {"name": "attention_8x16x8192x128", "kind": "attention", "dtype": "float16", "batch": 8, "heads": 16, "seq": 8192,
         "dim": 128, "causal": False, "padded": False},
        # the fp32 drop-in binding on one odd-length sequence with padding
        {"name": "attention_f32_1x12x197x64", "kind": "attention", "dtype": "float32", "batch": 1, "heads": 12, "seq": 197,
         "dim": 64, "causal": False, "padded": True},
        # the fp32 drop-in matmul at a ragged size
        {"name": "matmul_f32_500x1000x768", "kind": "matmul", "dtype": "float32", "m": 500, "n": 1000, "k": 768},
        # residual + LayerNorm with the int8 copy, as a model built from the operators calls it
        {"name": "add_layernorm_12288x1024", "kind": "rowwise", "op": "add_layernorm", "rows": 12288, "hidden": 1024},
    ]


def _log_int(rng, lo, hi):
    """Log-uniform over lo .. hi."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choices(("encoder", "attention", "linear", "matmul", "rowwise"), (9, 3, 2, 1, 1))[0]
    if kind == "encoder":
        precision = rng.choices(("int8", "fp16"), (3, 1))[0]
        model = rng.choices(("base", "large"), (3, 1))[0]
        form = rng.choices(("forward", "replay", "host", "unpadded"), (3, 4, 2, 2))[0]
        seq = rng.randint(65, 512) if form == "unpadded" else _log_int(rng, 8, 512)
        # no more work than the large model's shard (a stream of host batches is several passes)
        most = 32 * 384 * (1.0 if model == "large" else 3.5) / (2 if precision == "fp16" else 1) / (HOST_BATCHES if form == "host" else 1)
        batch = _log_int(rng, 4 if form == "unpadded" else 1, max(4, min(128, int(most // seq))))
        return {"kind": "encoder", "precision": precision, "model": model, "batch": batch, "seq": seq, "form": form}
    if kind == "attention":
        dtype = rng.choices(("float16", "float32"), (3, 1))[0]
        dim, batch, heads = rng.choice((64, 128)), _log_int(rng, 1, 16), rng.choice((8, 12, 16))
        longest = int(math.sqrt(8 * 16 * 8192.0**2 * 128 / (batch * heads * dim)))
        seq = _log_int(rng, 16, min(8192 if dtype == "float16" else 1024, longest))
        return {"kind": "attention", "dtype": dtype, "batch": batch, "heads": heads, "seq": seq, "dim": dim,
                "causal": rng.random() < 0.4, "padded": rng.random() < 0.4}
    if kind == "linear":
        n, k = rng.choice(PROJECTIONS)
        precision = rng.choice(("int8", "fp16"))
        return {"kind": "linear", "precision": precision, "m": _log_int(rng, 1, 16384), "n": n, "k": k,
                "act": rng.choice(("none", "gelu")), "out": rng.choice(("float32", "float16", "int8") if precision == "int8" else ("float16",))}
    if kind == "matmul":
        # rows of any number; K (and N for fp16 operands) in the 16-byte units that the operands need
        dtype = rng.choice(("float32", "float16"))
        n = _log_int(rng, 16, 4096)
        return {"kind": "matmul", "dtype": dtype, "m": _log_int(rng, 16, 4096), "n": n if dtype == "float32" else -(-n // 8) * 8,
                "k": -(-_log_int(rng, 16, 4096) // 8) * 8}
    return {"kind": "rowwise", "op": rng.choice(("layernorm", "add_layernorm", "gelu")), "rows": _log_int(rng, 1, 32768),
            "hidden": rng.choice((384, 768, 1000, 1024, 3072))}


# ---------------------------------------------------------------------------------------------
# what a program has in hand before the call
# ---------------------------------------------------------------------------------------------
class _Rand:
    """Seeded values made on the device."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEVICE).manual_seed(int(seed))

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.float32):
        x = torch.randn(shape, generator=self.g, device=DEVICE, dtype=torch.float32)
        return x.mul_(std).add_(mean).to(dtype)

    def int8(self, *shape):
        """Weights N(0, s) at the per-channel scale absmax / 127.5, absmax a little over three standard deviations."""
        return self.normal(*shape, std=38.0).round_().clamp_(-127, 127).to(torch.int8)

    def ints(self, lo, hi, *shape):
        return torch.randint(lo, hi, shape, generator=self.g, device=DEVICE, dtype=torch.int32)


def _host(t):
    return t.cpu().numpy()


def _encoder_params(r, cfg, precision):
    H, F = cfg.hidden, cfg.ffn
    p = {"word": _host(r.normal(cfg.vocab, H, std=0.02)), "pos": _host(r.normal(cfg.max_pos, H, std=0.02)),
         "type": _host(r.normal(cfg.type_vocab, H, std=0.02)), "emb_ln_g": _host(r.normal(H, std=0.1, mean=1.0)),
         "emb_ln_b": _host(r.normal(H, std=0.1)), "layers": []}
    shapes = {"wqkv": (3 * H, H), "wo": (H, H), "w1": (F, H), "w2": (H, F)}
    weights = []
    for _ in range(cfg.layers):
        lp = {b: _host(r.normal(n, std=0.02)) for b, n in (("bqkv", 3 * H), ("bo", H), ("b1", F), ("b2", H))}
        for n in ("ln1", "ln2"):
            lp[n + "_g"], lp[n + "_b"] = _host(r.normal(H, std=0.1, mean=1.0)), _host(r.normal(H, std=0.1))
        if precision == "fp16":
            lp.update({k: _host(r.normal(*s, std=0.02)) for k, s in shapes.items()})
        else:
            weights.append({k: (_host(r.int8(*s)), _host(r.normal(s[0], std=2e-5, mean=5.2e-4))) for k, s in shapes.items()})
        p["layers"].append(lp)
    act = [{"x": 0.036, "ctx": 0.012, "h1": 0.036, "gelu": 0.022} for _ in range(cfg.layers)]
    return p, Int8Scales(act=act, weights=weights)


def _key_lens(r, case):
    B, S = case["batch"], case["seq"]
    if case.get("form") == "unpadded":
        return S - r.ints(0, S - S // 4 + 1, B)  # documents of a quarter to all of the length
    return S - r.ints(0, min(32, S // 4) + 1, B)


def _prepare_encoder(case, r):
    cfg = MODELS[case["model"]]
    B, S, form = case["batch"], case["seq"], case["form"]
    params, scales = _encoder_params(r, cfg, case["precision"])
    enc = Fp16Encoder(cfg, params, DEVICE) if case["precision"] == "fp16" else Int8Encoder(cfg, params, scales, DEVICE)
    batches = [(r.ints(0, cfg.vocab, B, S), _key_lens(r, case)) for _ in range(HOST_BATCHES if form == "host" else 1)]
    st = {"form": form, "enc": enc}
    if form == "host":
        st["pipe"] = HostPipeline(enc, B, S, depth=HOST_BATCHES)
        st["batches"] = [(i.cpu().pin_memory(), n.cpu().pin_memory()) for i, n in batches]
        return st
    st["ids"], st["lens"] = batches[0]
    if form == "replay":
        enc.capture(B, S)
    elif form == "unpadded":
        enc.capture_unpadded(B, S, enc.unpadded_capacity(st["lens"].tolist(), S))
    return st


def _prepare_attention(case, r):
    shape = (case["batch"], case["heads"], case["seq"], case["dim"])
    dt = getattr(torch, case["dtype"])
    q, k, v = (r.normal(*shape, dtype=dt) for _ in range(3))
    return {"q": q, "k": k, "v": v, "causal": case["causal"], "lens": _key_lens(r, case) if case["padded"] else None}


def _prepare_linear(case, r):
    M, N, K = case["m"], case["n"], case["k"]
    st = {"precision": case["precision"], "act": case["act"], "out": getattr(torch, case["out"]), "bias": r.normal(N, std=0.02)}
    if case["precision"] == "int8":
        st.update(x=r.normal(M, K), x_scale=0.036, w=r.int8(N, K), w_scale=r.normal(N, std=2e-5, mean=5.2e-4), out_scale=0.022)
    else:
        st.update(x=r.normal(M, K, dtype=torch.float16), w=r.normal(N, K, std=0.02, dtype=torch.float16))
    return st


def _prepare_matmul(case, r):
    dt = getattr(torch, case["dtype"])
    return {"a": r.normal(case["m"], case["k"], dtype=dt), "b": r.normal(case["k"], case["n"], dtype=dt)}


def _prepare_rowwise(case, r):
    dt = torch.float16 if case["op"] == "add_layernorm" else torch.float32
    R, H = case["rows"], case["hidden"]
    return {"op": case["op"], "x": r.normal(R, H, dtype=dt), "residual": r.normal(R, H, dtype=dt) if case["op"] == "add_layernorm" else None,
            "gamma": r.normal(H, std=0.1, mean=1.0, dtype=dt), "beta": r.normal(H, std=0.1, dtype=dt)}


_PREPARE = {"encoder": _prepare_encoder, "attention": _prepare_attention, "linear": _prepare_linear, "matmul": _prepare_matmul,
            "rowwise": _prepare_rowwise}


def prepare(case, seed):
    st = _PREPARE[case["kind"]](case, _Rand(seed))
    st["kind"] = case["kind"]
    return st


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
def _run_encoder(st):
    enc, form = st["enc"], st["form"]
    if form == "host":
        tickets = [st["pipe"].submit(ids, lens) for ids, lens in st["batches"]]
        return [st["pipe"].result(t) for t in tickets]
    if form == "forward":
        return enc.forward(st["ids"], st["lens"])
    enc.set_inputs(st["ids"], st["lens"])
    return enc.replay()


def _run_attention(st):
    return zenith_cuda.flash_attention(st["q"], st["k"], st["v"], causal=st["causal"], kv_lens=st["lens"])


def _run_linear(st):
    if st["precision"] == "fp16":
        return ops.linear_fp16(st["x"], st["w"], st["bias"], act=st["act"], out_dtype=st["out"])
    xq = ops.quantize(st["x"], st["x_scale"])
    y = ops.linear_int8(xq, st["w"], st["x_scale"], st["w_scale"], st["bias"], act=st["act"], out_dtype=st["out"],
                        out_scale=st["out_scale"] if st["out"] == torch.int8 else None)
    return xq, y


def _run_matmul(st):
    return (zenith_cuda.matmul if st["a"].dtype == torch.float32 else zenith_cuda.wmma_matmul)(st["a"], st["b"])


def _run_rowwise(st):
    if st["op"] == "gelu":
        return zenith_cuda.gelu(st["x"])
    if st["op"] == "layernorm":
        return zenith_cuda.layernorm(st["x"], st["gamma"], st["beta"], 1e-12)
    return ops.add_layernorm(st["x"], st["residual"], st["gamma"], st["beta"], 1e-12, out_scale=0.036)


_RUN = {"encoder": _run_encoder, "attention": _run_attention, "linear": _run_linear, "matmul": _run_matmul, "rowwise": _run_rowwise}


def run(state):
    return _RUN[state["kind"]](state)


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without, and how close another correct implementation comes
# ---------------------------------------------------------------------------------------------
def _mean_len(case):
    S = case["seq"]
    return S - (0.375 * S if case.get("form") == "unpadded" else min(32, S // 4) / 2)


def work(case):
    kind = case["kind"]
    if kind == "encoder":
        cfg = MODELS[case["model"]]
        B, S, H, F, L = case["batch"], case["seq"], cfg.hidden, cfg.ffn, cfg.layers
        n = _mean_len(case)
        rows, q = (n, n) if case["form"] == "unpadded" else (S, S)
        passes = HOST_BATCHES if case["form"] == "host" else 1
        elem = 2 if case["precision"] == "fp16" else 1
        weights = L * (4 * H * H + 2 * H * F)
        flops = 2 * B * rows * weights + L * 4 * B * q * n * H
        data = min(B * rows, cfg.vocab) * H * 2 + 4 * B * (S + 1) + B * S * H * 2
        return {"bytes": weights * elem + passes * data, "flops": passes * flops}
    if kind == "attention":
        B, H, S, D = case["batch"], case["heads"], case["seq"], case["dim"]
        n = _mean_len(case) if case["padded"] else S
        pairs = S * n - n * (n - 1) / 2 if case["causal"] else S * n
        return {"bytes": 4 * B * H * S * D * (2 if case["dtype"] == "float16" else 4), "flops": 4 * B * H * D * pairs}
    if kind in ("linear", "matmul"):
        M, N, K = case["m"], case["n"], case["k"]
        if kind == "matmul":
            a, o = (4, 4) if case["dtype"] == "float32" else (2, 4)
            return {"bytes": a * (M * K + K * N) + o * M * N, "flops": 2 * M * N * K}
        o = {"float32": 4, "float16": 2, "int8": 1}[case["out"]]
        x, w = (2, 2) if case["precision"] == "fp16" else (5, 1)  # the int8 form reads fp32 activations and returns their int8 copy
        return {"bytes": x * M * K + w * N * K + 8 * N + o * M * N, "flops": 2 * M * N * K}
    R, H = case["rows"], case["hidden"]
    return {"bytes": R * H * {"gelu": 8, "layernorm": 8, "add_layernorm": 7}[case["op"]], "flops": R * H * 10}


def tolerance(case):
    kind = case["kind"]
    if kind == "encoder":
        # fp16 roundings that add up over the layers; with int8 operands they also move values across rounding boundaries
        return {"rel": 5e-3 if case["precision"] == "int8" else 3e-3}
    if kind == "attention":
        return {"rel": 2e-3}  # fp16 operands, probabilities and result (the fp32 binding computes in fp16 too)
    if kind == "linear":
        if case["precision"] == "fp16":
            return {"rel": 1e-3}
        return "exact" if case["out"] == "int8" else {"rel": 1e-3 if case["out"] == "float16" else 1e-6}
    if kind == "matmul":
        return {"rel": 1e-3 if case["dtype"] == "float32" else 1e-5}  # TF32 / fp16 operands, fp32 sums
    if case["op"] == "add_layernorm":
        return {"rel": 2e-3, "differ": 2e-3}  # fp16 result, and an int8 copy that follows its roundings
    return {"rel": 1e-5}

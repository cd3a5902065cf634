"""The work that users of this framework have it do, as cases that can be timed.

Every case goes through the public classes (`TurboQuantV3`, `MSECompressor`, `TurboQuantCompressorV2`,
`TurboQuantKVCache`, `V3Cache`, `batched.CachePlan`) on synthetic K/V: N(0, 1) entries with 4 channels in 128 per
head scaled by 10, as the caches that this format is made for look.  The codecs (rotation matrices, codebooks and the
kernel-side constants made from them) belong to a model's layer, not to its inputs: a program builds them once, and so
does this file.
"""

import functools
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "turboquant-pytorch_b200"))

from turboquant import MSECompressor, TurboQuantCompressorV2, TurboQuantKVCache, TurboQuantV3, batched, cache  # noqa: E402

DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}
DEVICE = "cuda"
MAX_LAYERS = 10


def listed():
    return [
        # a short prompt of a small GQA model (2 KV heads), one layer through compress_kv and decompress_kv: 172 tokens
        # leave the window.  Launches and host work are all there is
        {"name": "layer_short", "kind": "layer", "batch": 1, "heads": 2, "seq": 300, "dim": 128, "dtype": "fp16",
         "key_bits": 4, "value_bits": 2, "window": 128},
        # one layer of the Qwen2.5-3B-shaped cache (2 KV heads, 8192 tokens, K4/V2, no window)
        {"name": "layer_8k", "kind": "layer", "batch": 1, "heads": 2, "seq": 8192, "dim": 128, "dtype": "fp16",
         "key_bits": 4, "value_bits": 2, "window": 0},
        # head_dim 64, a ragged length and 3-bit codes, as smaller models have them
        {"name": "layer_dim64", "kind": "layer", "batch": 2, "heads": 8, "seq": 5003, "dim": 64, "dtype": "bf16",
         "key_bits": 4, "value_bits": 3, "window": 128},
        # a slice of the Llama-3-8B-shaped cache: 8 layers, the first and the last protected with 8 bits, K6/V4
        # elsewhere, 128 tokens kept: compress and decompress of a whole cache in static buffers
        {"name": "cache_32k", "kind": "cache", "layers": 8, "batch": 4, "heads": 8, "seq": 32768, "dim": 128,
         "dtype": "bf16", "key_bits": 6, "value_bits": 4, "window": 128, "protected": 1},
        # 4096 fp32 vectors through one codec and back, the reference's basic round trip
        {"name": "mse_fp32", "kind": "mse", "batch": 1, "heads": 1, "seq": 4096, "dim": 128, "dtype": "fp32", "bits": 4},
        # one token for every layer of a model that is generating: each layer quantises the token that leaves its
        # window.  What it costs does not depend on the tokens that are there already
        {"name": "cache_step", "kind": "step", "layers": 32, "batch": 1, "heads": 8, "seq": 512, "dim": 128,
         "dtype": "bf16", "key_bits": 6, "value_bits": 4, "window": 128},
        # logits and softmax straight from 131072 packed 4-bit keys per head, 32 query heads on 8 KV heads
        {"name": "packed_scores", "kind": "scores", "batch": 1, "heads": 8, "q_heads": 32, "queries": 1, "seq": 131072,
         "dim": 128, "dtype": "fp16", "bits": 4},
        # decode attention of one token from packed K4/V2 and the kept window
        {"name": "decode_attention", "kind": "decode", "batch": 1, "heads": 8, "q_heads": 32, "queries": 1,
         "seq": 32768, "dim": 128, "dtype": "fp16", "key_bits": 4, "value_bits": 2, "window": 128},
        # the MSE + QJL form of 16 heads x 16384 keys of head_dim 256 at 3 bits, in the reference's layout
        {"name": "qjl_compress", "kind": "v2_compress", "batch": 1, "heads": 16, "seq": 16384, "dim": 256,
         "dtype": "fp16", "bits": 3, "packed": False},
        # scores of 64 queries per head against those keys
        {"name": "qjl_scores", "kind": "v2_scores", "batch": 1, "heads": 16, "queries": 64, "seq": 16384, "dim": 256,
         "dtype": "fp16", "bits": 3, "packed": False},
        # the bit-packed storage of the same representation at head_dim 128, compressed and scored in one pass
        {"name": "qjl_packed", "kind": "v2_both", "batch": 1, "heads": 8, "queries": 16, "seq": 4096, "dim": 128,
         "dtype": "fp16", "bits": 3, "packed": True},
        # the first-generation cache: 8192 unit keys and values appended, scored by one query and read back
        {"name": "v1_cache", "kind": "v1", "seq": 8192, "dim": 128, "bits": 3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shrink(case, most):
    """Shortens `seq` until the case has at most `most` vectors per tensor."""
    per = case.get("batch", 1) * case.get("heads", 1) * case.get("layers", 1)
    case["seq"] = max(case.get("window", 0) + 1, min(case["seq"], most // per))
    return case


def draw(rng):
    kind = rng.choice(["layer", "layer", "layer", "cache", "cache", "mse", "step", "scores", "scores", "decode", "decode",
                       "v2_compress", "v2_scores", "v2_both", "v1"])
    pair = rng.choice([(4, 2), (4, 2), (6, 4), (6, 4), (4, 4), (3, 3), (8, 8)])
    half = rng.choice(["fp16", "bf16"])
    window = rng.choice([0, 128])
    heads = rng.choice([2, 4, 8])
    batch = rng.choice([1, 1, 2, 4])
    if kind == "layer":
        return _shrink({"kind": kind, "batch": batch, "heads": heads, "seq": window + _log_int(rng, 100, 32768),
                        "dim": rng.choice([128, 128, 128, 64]), "dtype": half, "key_bits": pair[0], "value_bits": pair[1],
                        "window": window}, 1 << 20)
    if kind == "cache":
        return _shrink({"kind": kind, "layers": rng.randint(4, MAX_LAYERS), "batch": batch, "heads": heads,
                        "seq": window + _log_int(rng, 1000, 32768), "dim": 128, "dtype": half, "key_bits": pair[0],
                        "value_bits": pair[1], "window": window, "protected": rng.choice([0, 1])}, 8 << 20)
    if kind == "mse":
        return _shrink({"kind": kind, "batch": batch, "heads": rng.choice([1, heads]), "seq": _log_int(rng, 64, 16384),
                        "dim": rng.choice([128, 128, 64]), "dtype": rng.choice(["fp32", "fp32", half]),
                        "bits": rng.choice([2, 3, 4, 4, 6, 8])}, 1 << 18)
    if kind == "step":
        return {"kind": kind, "layers": rng.choice([16, 24, 28, 32]), "batch": rng.choice([1, 1, 2]), "heads": heads,
                "seq": window + rng.randint(1, 500), "dim": 128, "dtype": half, "key_bits": pair[0],
                "value_bits": pair[1], "window": window}
    if kind == "scores":
        return _shrink({"kind": kind, "batch": batch, "heads": heads, "q_heads": heads * rng.choice([1, 4, 4, 8]),
                        "queries": rng.choice([1, 1, 1, 4]), "seq": _log_int(rng, 500, 131072), "dim": 128, "dtype": half,
                        "bits": rng.choice([2, 4, 4, 6, 8])}, 1 << 20)
    if kind == "decode":
        return _shrink({"kind": kind, "batch": batch, "heads": heads, "q_heads": heads * rng.choice([1, 4, 4, 8]),
                        "queries": 1, "seq": window + _log_int(rng, 500, 131072), "dim": 128, "dtype": half,
                        "key_bits": pair[0], "value_bits": pair[1], "window": window}, 1 << 20)
    if kind == "v1":
        return {"kind": kind, "seq": _log_int(rng, 500, 16384), "dim": rng.choice([64, 128, 128]),
                "bits": rng.choice([2, 3, 4])}
    return _shrink({"kind": kind, "batch": batch, "heads": rng.choice([2, 8, 16]), "queries": rng.choice([1, 16, 64]),
                    "seq": _log_int(rng, 256, 16384), "dim": rng.choice([128, 256]), "dtype": "fp16",
                    "bits": rng.choice([2, 3, 3, 4]), "packed": rng.choice([True, False])}, 1 << 18)


# ------------------------------------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _kv(gen, batch, heads, seq, dim, dtype):
    """(B, H, S, D) entries N(0, 1), 4 of every 128 channels of a head scaled by 10."""
    x = torch.randn(batch, heads, seq, dim, generator=gen, device=DEVICE)
    hot = torch.rand(heads, dim, generator=gen, device=DEVICE).argsort(dim=1) < 4 * dim // 128
    x *= torch.where(hot, 10.0, 1.0)[None, :, None, :]
    return x.to(DTYPES[dtype])


@functools.lru_cache(maxsize=None)
def _layer_codec(dim, key_bits, value_bits, window, layer, n_layers, protected):
    return TurboQuantV3(dim, key_bits=key_bits, value_bits=value_bits, residual_window=window, layer_idx=layer,
                        n_layers=n_layers, protected_layers=protected, device=DEVICE)


@functools.lru_cache(maxsize=None)
def _mse_codec(dim, bits):
    return MSECompressor(dim, bits, seed=42, device=DEVICE)


@functools.lru_cache(maxsize=None)
def _v2_codec(dim, bits):
    return TurboQuantCompressorV2(dim, bits, seed=42, device=DEVICE)


def _codec(case, layer=0):
    return _layer_codec(case["dim"], case["key_bits"], case["value_bits"], case["window"], layer,
                        case.get("layers", 1), case.get("protected", 0))


def prepare(case, seed):
    kind, gen = case["kind"], _generator(seed)
    state = {"case": case}
    if kind == "v1":
        state["cache"] = TurboQuantKVCache(case["dim"], case["dim"], bits=case["bits"], device=DEVICE)
        for name, rows in (("keys", case["seq"]), ("values", case["seq"]), ("query", 1)):
            x = torch.randn(rows, case["dim"], generator=gen, device=DEVICE)
            state[name] = x / x.norm(dim=-1, keepdim=True)
        return state
    shape = (case["batch"], case["heads"], case["seq"], case["dim"])
    if kind in ("layer", "decode"):
        state["codec"] = _codec(case)
        state["keys"], state["values"] = (_kv(gen, *shape, case["dtype"]) for _ in range(2))
    elif kind == "cache":
        keys, values = ([_kv(gen, *shape, case["dtype"]) for _ in range(case["layers"])] for _ in range(2))
        state["plan"] = batched.CachePlan([_codec(case, l) for l in range(case["layers"])], keys, values)
        state["inputs"] = keys, values
    elif kind in ("mse", "scores"):
        state["codec"] = _mse_codec(case["dim"], case["bits"])
        state["keys"] = _kv(gen, *shape, case["dtype"])
    elif kind == "step":
        # a cache that has seen its prompt, with room for the tokens to come
        c = cache.V3Cache(key_bits=case["key_bits"], value_bits=case["value_bits"], residual_window=case["window"],
                          n_layers=case["layers"], initial_capacity=16384)
        for l in range(case["layers"]):
            c.update(_kv(gen, *shape, case["dtype"]), _kv(gen, *shape, case["dtype"]), l)
        token = (case["batch"], case["heads"], 1, case["dim"])
        state["cache"] = c
        state["keys"], state["values"] = ([_kv(gen, *token, case["dtype"]) for _ in range(case["layers"])] for _ in range(2))
    else:
        state["codec"] = _v2_codec(case["dim"], case["bits"])
        state["keys"] = _kv(gen, *shape, case["dtype"])
    if "queries" in case:
        state["queries"] = torch.randn(case["batch"], case.get("q_heads", case["heads"]), case["queries"], case["dim"],
                                       generator=gen, device=DEVICE).to(DTYPES[case["dtype"]])
    # attention reads what an earlier call has packed; these bytes are inputs, so they come from the seed and not from
    # the kernels that are timed in other cases
    if kind == "scores":
        state["packed"] = _mse_form(state.pop("keys"), state["codec"])
    elif kind == "decode":
        state["packed"] = tuple(_window_form(state[name], codec, case["window"]) for name, codec in _sides(state["codec"]))
    elif kind == "v2_scores":
        state["packed"] = _v2_form(state.pop("keys"), state["codec"], case["packed"])
    return state


# ------------------------------------------------------------------------------------------------ the formats in 64 bits
def _sides(codec):
    return ("keys", codec.key_compressor), ("values", codec.val_compressor)


def _indices(y, centroids):
    c = centroids.double()
    return torch.searchsorted((c[1:] + c[:-1]) / 2, y)


def _quantise(x, pi, centroids, normalise=True):
    """(indices, norms) of 64-bit vectors; the first or last index for what lies outside."""
    norms = x.norm(dim=-1)
    unit = x / (norms + 1e-8).unsqueeze(-1) if normalise else x
    return _indices(unit @ pi.double().T, centroids), norms


def _pack(idx, bits):
    per = 8 // bits
    fields = idx.reshape(*idx.shape[:-1], -1, per)
    out = torch.zeros(fields.shape[:-1], dtype=torch.int64, device=idx.device)
    for i in range(per):
        out |= fields[..., i] << (bits * (per - 1 - i))
    return out.to(torch.uint8)


def _unpack(packed, bits):
    per = 8 // bits
    fields = [(packed.long() >> (bits * (per - 1 - i))) & ((1 << bits) - 1) for i in range(per)]
    return torch.stack(fields, dim=-1).flatten(-2)


def _mse_form(x, codec):
    idx, norms = _quantise(x.double(), codec.Pi, codec.centroids)
    return {"idx_bytes": _pack(idx, codec.bits), "vec_norms": norms.half(), "shape": tuple(x.shape), "idx_pad": 0}


def _window_form(x, codec, window):
    cut = x.shape[2] - window
    return {"compressed": _mse_form(x[:, :, :cut], codec), "fp16": x[:, :, cut:], "shape": tuple(x.shape), "split_at": cut}


def _mse_back(packed, codec):
    levels = codec.centroids.double()[_unpack(packed["idx_bytes"], codec.bits)]
    return (levels @ codec.Pi.double()) * packed["vec_norms"].double().unsqueeze(-1)


def _window_back(packed, codec):
    return torch.cat([_mse_back(packed["compressed"], codec), packed["fp16"].double()], dim=2)


def _residual(x, pi, centroids, s, normalise=True):
    """(indices, norms, MSE reconstruction, residual norms, signs) of the MSE + QJL form."""
    idx, norms = _quantise(x, pi, centroids, normalise)
    mse = centroids.double()[idx] @ pi.double()
    if normalise:
        mse = mse * norms.unsqueeze(-1)
    rest = x - mse
    return idx, norms, mse, rest.norm(dim=-1), torch.where(rest @ s.double().T >= 0, 1.0, -1.0).double()


def _v2_form(x, codec, packed):
    idx, norms, mse, rnorm, signs = _residual(x.double(), codec.Pi, codec.centroids, codec.S)
    if not packed:
        return {"k_mse": mse.half(), "qjl_signs": signs.to(torch.int8), "residual_norm": rnorm.half(), "shape": tuple(x.shape)}
    return {"mse_idx_bytes": _pack(idx, codec.mse_bits), "sign_bits": _pack((signs > 0).long(), 1), "vec_norms": norms.float(),
            "residual_norm": rnorm.half(), "shape": tuple(x.shape), "packed": True}


def _v2_scores(q, packed, codec):
    if packed.get("packed"):
        levels = codec.centroids.double()[_unpack(packed["mse_idx_bytes"], codec.mse_bits)]
        mse = (levels @ codec.Pi.double()) * packed["vec_norms"].double().unsqueeze(-1)
        signs = _unpack(packed["sign_bits"], 1).double() * 2 - 1
    else:
        mse, signs = packed["k_mse"].double(), packed["qjl_signs"].double()
    corr = math.sqrt(math.pi / 2) / q.shape[-1] * packed["residual_norm"].double().unsqueeze(-2)
    return q @ mse.transpose(-1, -2) + (q @ codec.S.double().T) @ signs.transpose(-1, -2) * corr


def exact(case, seed):
    """What `run` returns, from 64-bit sums.  None stands for indices and signs: those are right or wrong, not near."""
    kind = case["kind"]
    vectors = case.get("layers", 1) * case.get("batch", 1) * case.get("heads", 1) * case["seq"]
    if kind == "cache" and vectors > 1 << 20:
        return None
    if kind == "step":
        gen = _generator(seed)
        token = (case["batch"], case["heads"], 1, case["dim"])
        shape = (case["batch"], case["heads"], case["seq"], case["dim"])
        whole = [[_kv(gen, *shape, case["dtype"]) for _ in range(2)] for _ in range(case["layers"])]
        new = [[_kv(gen, *token, case["dtype"]) for _ in range(case["layers"])] for _ in range(2)]
        out = []
        for l, pair in enumerate(whole):
            codec = _layer_codec(case["dim"], case["key_bits"], case["value_bits"], 0, l, case["layers"], 0)
            out.append(tuple(_window_back(_window_form(torch.cat([x, new[i][l]], dim=2), side, case["window"]), side)
                             for i, (x, (_, side)) in enumerate(zip(pair, _sides(codec)))))
        return out
    state = prepare(case, seed)
    if kind in ("layer", "cache"):
        inputs = [state["keys"]], [state["values"]]
        if kind == "cache":
            inputs = state["inputs"]
        out = []
        for l in range(case.get("layers", 1)):
            forms, back = [], []
            for x, (_, side) in zip((inputs[0][l], inputs[1][l]), _sides(_codec(case, l))):
                form = _window_form(x, side, case["window"])
                cut = form["split_at"]
                forms.append({"idx_bytes": None, "vec_norms": x[:, :, :cut].double().norm(dim=-1)})
                back.append(_window_back(form, side))
            out.append(forms + back)
        return out if kind == "cache" else dict(zip(("k", "v", "keys", "values"), out[0]))
    if kind == "mse":
        form = _mse_form(state["keys"], state["codec"])
        return {"packed": {"idx_bytes": None, "vec_norms": state["keys"].double().norm(dim=-1)},
                "keys": _mse_back(form, state["codec"])}
    if kind == "v1":
        key, value = state["cache"].key_quantizer, state["cache"].value_quantizer
        _, _, mse, rnorm, signs = _residual(state["keys"].double(), key.mse.Pi, key.mse.centroids, key.S, normalise=False)
        q = state["query"].double()
        scores = q @ mse.T + math.sqrt(math.pi / 2) / case["dim"] * rnorm * ((q @ key.S.double().T) @ signs.T)
        idx, _ = _quantise(state["values"].double(), value.Pi, value.centroids, normalise=False)
        return {"k": {"mse_indices": None, "qjl_signs": None, "residual_norm": rnorm}, "v": None, "scores": scores[0],
                "values": value.centroids.double()[idx] @ value.Pi.double()}
    queries, codec = state.get("queries"), state["codec"]
    if kind in ("scores", "decode"):
        group = case["q_heads"] // case["heads"]
        back = _mse_back(state["packed"], codec) if kind == "scores" else _window_back(state["packed"][0], codec.key_compressor)
        q = queries.double().unflatten(1, (case["heads"], group)).flatten(2, 3)
        logits = q @ back.transpose(-1, -2) * case["dim"] ** -0.5
        lead = (case["batch"], case["q_heads"], case["queries"], -1)
        probs = logits.softmax(dim=-1)
        if kind == "scores":
            return logits.reshape(lead), probs.reshape(lead)
        return (probs @ _window_back(state["packed"][1], codec.val_compressor)).reshape(lead)
    if kind == "v2_scores":
        return _v2_scores(queries.double(), state["packed"], codec)
    form = _v2_form(state["keys"], codec, case["packed"])
    _, norms, mse, rnorm, _ = _residual(state["keys"].double(), codec.Pi, codec.centroids, codec.S)
    if case["packed"]:
        out = {"mse_idx_bytes": None, "sign_bits": None, "vec_norms": norms, "residual_norm": rnorm}
    else:
        out = {"k_mse": mse, "qjl_signs": None, "residual_norm": rnorm}
    if kind == "v2_compress":
        return out
    return {"packed": out, "scores": _v2_scores(queries.double(), form, codec)}


def _tensors(compressed):
    """The tensors of what compress / compress_kv returned."""
    if isinstance(compressed, dict):
        return {k: _tensors(v) for k, v in compressed.items() if isinstance(v, (dict, torch.Tensor))}
    return compressed


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "layer":
        ck, cv = state["codec"].compress_kv(state["keys"], state["values"])
        keys, values = state["codec"].decompress_kv(ck, cv)
        return {"k": _tensors(ck["compressed"]), "v": _tensors(cv["compressed"]), "keys": keys, "values": values}
    if kind == "cache":
        packed = state["plan"].compress()
        full = state["plan"].decompress()
        return [[_tensors(ck["compressed"]), _tensors(cv["compressed"]), keys, values]
                for (ck, cv), (keys, values) in zip(packed, full)]
    if kind == "mse":
        packed = state["codec"].compress(state["keys"])
        return {"packed": _tensors(packed), "keys": state["codec"].decompress(packed)}
    if kind == "step":
        return state["cache"].step(state["keys"], state["values"])
    if kind == "scores":
        return state["codec"].attention_scores(state["queries"], state["packed"], scale=case["dim"] ** -0.5, softmax=True)
    if kind == "decode":
        return state["codec"].decode_attention(state["queries"], *state["packed"])
    if kind == "v1":
        c = state["cache"]
        c.key_cache.clear()
        c.value_cache.clear()
        c.append(state["keys"], state["values"])
        key, value = c.key_cache[0], c.value_cache[0]
        return {"k": _tensors(key), "v": value["indices"], "scores": c.attention_scores(state["query"]), "values": c.get_values()}
    codec = state["codec"]
    if kind == "v2_compress":
        return _tensors(codec.compress(state["keys"], packed=case["packed"]))
    if kind == "v2_scores":
        return codec.asymmetric_attention_scores(state["queries"], state["packed"])
    packed = codec.compress(state["keys"], packed=case["packed"])
    return {"packed": _tensors(packed), "scores": codec.asymmetric_attention_scores(state["queries"], packed)}


# ------------------------------------------------------------------------------------------------ sizes and tolerances
def _row_bytes(dim, bits):
    return -(-dim // (8 // bits))


def _layer_bits(case, layer):
    guarded = layer < case.get("protected", 0) or layer >= case.get("layers", 1) - case.get("protected", 0)
    return (8, 8) if guarded and case.get("protected", 0) else (case["key_bits"], case["value_bits"])


def work(case):
    """Bytes and operations of one pass.  A rotation of a vector is 2 D^2 operations."""
    kind, d, s = case["kind"], case["dim"], case["seq"]
    rows = case.get("batch", 1) * case.get("heads", 1)
    elem = 4 if case.get("dtype", "fp32") == "fp32" else 2
    if kind in ("layer", "cache"):
        # 16-bit tensors in, packed rows and norms out and in again, 16-bit tensors out (the window with them)
        n, tokens = rows * (s - case["window"]), rows * s
        total = 0
        for l in range(case.get("layers", 1)):
            total += sum(2 * tokens * d * elem + 2 * n * (_row_bytes(d, b) + 2) for b in _layer_bits(case, l))
        return {"bytes": total, "flops": case.get("layers", 1) * 2 * 2 * n * 2 * d * d}
    if kind == "mse":
        n = rows * s
        return {"bytes": n * (d * elem + 2 * (_row_bytes(d, case["bits"]) + 2) + d * 4), "flops": 2 * n * 2 * d * d}
    if kind == "step":
        # per layer and K/V: the new token in and out, one token leaving the window, its packed row and reconstruction
        per = rows * case["layers"]
        return {"bytes": per * sum(4 * d * elem + _row_bytes(d, b) + 2 for b in (case["key_bits"], case["value_bits"])),
                "flops": per * 2 * 2 * 2 * d * d}
    if kind in ("scores", "decode"):
        q = case["batch"] * case["q_heads"] * case["queries"]
        if kind == "scores":
            return {"bytes": rows * s * (_row_bytes(d, case["bits"]) + 2) + q * d * elem + 2 * 4 * q * s,
                    "flops": 2 * q * s * d + 2 * q * d * d}
        n = s - case["window"]
        packed = sum(_row_bytes(d, b) + 2 for b in (case["key_bits"], case["value_bits"]))
        return {"bytes": rows * (n * packed + 2 * case["window"] * d * elem) + q * d * (elem + 4),
                "flops": 4 * q * s * d + 4 * q * d * d}
    if kind == "v1":
        # keys and values in; int64 indices of both, fp32 signs and residual norms out, and in again for the scores and values
        stored = s * (2 * d * 8 + d * 4 + 4)
        return {"bytes": 2 * s * d * 4 + 2 * stored + s * d * 4 + s * 4, "flops": (3 + 1 + 1 + 1) * s * 2 * d * d}
    n = rows * s
    stored = (_row_bytes(d, max(case["bits"] - 1, 1)) + d // 8 + 6) if case["packed"] else 3 * d + 2
    compress = {"bytes": n * (d * elem + stored), "flops": 3 * n * 2 * d * d}
    q = rows * case.get("queries", 0)
    scores = {"bytes": n * stored + q * d * elem + 4 * q * s, "flops": 2 * 2 * q * s * d + 2 * 2 * q * d * d}
    if kind == "v2_compress":
        return compress
    if kind == "v2_scores":
        return scores
    return {k: compress[k] + scores[k] for k in compress}


def tolerance(case):
    """About four times what each path differs by from itself with all its sums in 64 bits.

    16-bit outputs and norms round to 1.7e-3 (bf16).  A rotated value that lies on the boundary between two centroids
    takes either index: up to 8e-6 of the packed bytes and 7e-6 of the signs, by which a reconstruction's value moves up
    to 0.3 of its root mean square (a whole vector's relative error stays below 2e-3).  Scores from given packed
    keys have no ties: 2e-6, and 1e-5 in single values."""
    kind = case["kind"]
    if kind in ("scores", "decode", "v2_scores"):
        return {"rel": 1e-5, "max": 1e-4}
    # the share stands for four ties where an output is small
    values = case.get("batch", 1) * case.get("heads", 1) * (case["seq"] - case.get("window", 0)) * case["dim"] / 8
    ties = {"differ": min(0.009, max(4e-5, 4 / values)), "max": 0.9}
    if kind in ("layer", "cache", "step"):
        return {"rel": 6e-3, **ties}
    return {"rel": {"mse": 6e-3 if case.get("dtype") == "bf16" else 2e-3, "v1": 2e-3}.get(kind, 3e-3), **ties}

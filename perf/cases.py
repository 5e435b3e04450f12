"""Performance cases: the work a program has this package do, through its public entry points.

Seven kinds of work cover the package's two directions (packing keys and values, reading the packed cache):

  decode      ``omni_attn`` over a resident packed cache: one query token per user up to short prefills of many
  step        one turn of a serving loop on ``QuantizedKVCache``: append every user's new token, attend to all of it
  append      ``rotate_quantize_append`` of a chunk of new keys and values (prefill)
  bake        the two calls of an offline bake, ``rotate_queries`` and then ``quantize_heads``
  dequantize  ``dequantize_heads``, the codec's other direction
  calibrate   ``calibrate_per_group``, one codebook per kv head, before a bake
  host        ``HostDecodeStep``: query and result in page-locked host memory

Keys and values are N(0, 1); where a case says so, four channels of every row are eight times larger (what the rotation
is for) or one value in a hundred is ten times larger.  The packed caches are made by the package's own codec.
"""
import math

import torch

from omnistack_rs_b200.kernels.fused_attention import omni_attn, pair_v_rows
from omnistack_rs_b200.kernels.hadamard import rotate_queries
from omnistack_rs_b200.kernels.quantize import dequantize_heads, quantize_heads, rotate_quantize_append
from omnistack_rs_b200.quantization import calibrate_per_group
from omnistack_rs_b200.serving import HostDecodeStep, QuantizedKVCache

HEAD_DIM = 128
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
DTYPE_BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}
# 16-level Lloyd-Max levels of a unit Gaussian (what calibration of rotated N(0, 1) rows gives)
LEVELS = (-2.733, -2.069, -1.618, -1.256, -0.9424, -0.6568, -0.3881, -0.1284,
          0.1284, 0.3881, 0.6568, 0.9424, 1.256, 1.618, 2.069, 2.733)
KEY_BYTES = 140             # one key of one kv head in attention: K 64 + 8 + 4, V 64
ROW_BYTES = 76              # one packed row: 64 nibble bytes, 8 sign bytes, one fp32 norm

DECODE = dict(kind="decode", tokens=1, ragged=0.0, dtype="bf16", per_head=True, pair=False, rotated=False, lora_rank=0, outliers=False)


def listed():
    return [
        # one ranking query: 64 users with a short history each, no query grouping (the smallest call)
        dict(DECODE, name="rank_64x50", users=64, q_heads=8, kv_heads=8, keys=50),
        # the same query in the shape of the reference's benchmark: grouped heads, per-user adapters, V read from K's codes
        dict(DECODE, name="rank_adapters_64x50", users=64, q_heads=32, kv_heads=8, keys=50, lora_rank=16),
        # grouped-query decode over contexts of 1,024 to 8,192 keys, resident cache in its own (pair) layout
        dict(DECODE, name="gqa_256_ragged", users=256, q_heads=32, kv_heads=8, keys=8192, ragged=0.125, per_head=False,
             pair=True, outliers=True),
        # a slice of box-scale serving: one query per user, 32 ungrouped heads, 2,048 keys (the largest call)
        dict(DECODE, name="serve_2048x2048", users=2048, q_heads=32, kv_heads=32, keys=2048, per_head=False, pair=True),
        # few users with long contexts, rotation folded into the query and out of the result
        dict(DECODE, name="long_4x32768", users=4, q_heads=32, kv_heads=8, keys=32768, dtype="fp16", rotated=True),
        # short prefill / speculative verification: 32 query tokens per user share every key
        dict(DECODE, name="tokens_32_64x2048", users=64, q_heads=32, kv_heads=8, keys=2048, tokens=32, per_head=False, pair=True),
        # one turn of a serving loop at moderate size: append one token per user, then attend
        dict(kind="step", name="step_64x1500", users=64, q_heads=32, kv_heads=8, keys=1500, ragged=0.25, dtype="bf16", new_tokens=1),
        # prefill: 256 new tokens of K and V for each of 1,024 users, heavy-tailed activations
        dict(kind="append", name="prefill_1024x256", users=1024, kv_heads=8, new_tokens=256, dtype="bf16", per_head=False, v_signs=True),
        # offline bake of an odd length in fp32, rotation and codec as separate calls (the reference's own sequence)
        dict(kind="bake", name="bake_fp32_256x203", users=256, kv_heads=8, keys=203, dtype="fp32"),
        # reading a cache back to fp32
        dict(kind="dequantize", name="dequantize_128x1024", users=128, kv_heads=8, keys=1024, with_qjl=True),
        # codebooks of eight kv heads from 64 users x 50 tokens of each
        dict(kind="calibrate", name="calibrate_8x409600", groups=8, samples=409600),
        # serving with queries and results in host memory
        dict(kind="host", name="host_512x2048", users=512, q_heads=32, kv_heads=32, keys=2048, ragged=0.0, dtype="bf16"),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["decode"] * 6 + ["step", "append", "append", "bake", "dequantize", "calibrate", "host"])
    if kind == "calibrate":
        groups = rng.choice([1, 2, 4, 8, 16])
        return dict(kind=kind, groups=groups, samples=_log_int(rng, 1 << 12, 1 << 20))
    dtype = rng.choice(["bf16", "bf16", "fp16", "fp32"])
    kv_heads = rng.choice([1, 4, 8, 8, 32])
    if kind == "append":
        new_tokens = _log_int(rng, 1, 2048)
        users = _log_int(rng, 1, min(4096, (1 << 21) / (kv_heads * new_tokens) + 1))
        return dict(kind=kind, users=users, kv_heads=kv_heads, new_tokens=new_tokens, dtype=dtype,
                    per_head=rng.random() < 0.5, v_signs=rng.random() < 0.5)
    if kind in ("bake", "dequantize"):
        keys = _log_int(rng, 1, 4096)
        users = _log_int(rng, 1, min(2048, (1 << 20) / (kv_heads * keys) + 1))
        if kind == "bake":
            return dict(kind=kind, users=users, kv_heads=kv_heads, keys=keys, dtype=dtype)
        return dict(kind=kind, users=users, kv_heads=kv_heads, keys=keys, with_qjl=rng.random() < 0.7)
    group = rng.choice([1, 1, 3, 4, 4, 8]) if kv_heads < 32 else 1
    keys = _log_int(rng, 8, 32768)
    most = (1 << 29) / (kv_heads * keys * KEY_BYTES)
    ragged = rng.choice([0.0, 0.125, 0.5])
    if kind == "step":
        users = _log_int(rng, 1, max(1, min(512, most)))
        return dict(kind=kind, users=users, q_heads=kv_heads * group, kv_heads=kv_heads, keys=max(keys, 16), ragged=ragged or 0.5,
                    dtype=dtype, new_tokens=rng.choice([1, 1, 1, 4, 17]))
    if kind == "host":
        users = _log_int(rng, 1, max(1, min(1024, most)))
        return dict(kind=kind, users=users, q_heads=kv_heads * group, kv_heads=kv_heads, keys=keys, ragged=ragged, dtype=dtype)
    tokens = rng.choice([1, 1, 1, 1, _log_int(rng, 2, 8), _log_int(rng, 9, 64)])
    most = min(most, 1e11 / (4.0 * HEAD_DIM * kv_heads * group * tokens * keys))
    users = _log_int(rng, 1, max(1, min(2048, most)))
    lora_rank = rng.choice([8, 16, 32]) if tokens == 1 and keys <= 512 and users <= 256 and rng.random() < 0.4 else 0
    return dict(DECODE, users=users, q_heads=kv_heads * group, kv_heads=kv_heads, keys=keys, tokens=tokens, ragged=ragged, dtype=dtype,
                per_head=rng.random() < 0.5, pair=not lora_rank and rng.random() < 0.5, rotated=rng.random() < 0.3, lora_rank=lora_rank,
                outliers=rng.random() < 0.3)


# ---- inputs ---------------------------------------------------------------------------------------------------
def _rows(shape, gen, dtype, outliers=False, heavy=False):
    """Unrotated key or value rows."""
    x = torch.randn(shape, generator=gen, device="cuda", dtype=dtype)
    if outliers:
        x[..., [9, 40, 77, 102]] *= 8.0
    if heavy:
        x = torch.where(torch.rand(shape[:-1] + (HEAD_DIM,), generator=gen, device="cuda") < 0.01, x * 10.0, x)
    return x


def _codebooks(per_head, heads, scale=1.0):
    levels = torch.tensor(LEVELS, device="cuda") * scale
    if not per_head:
        return levels
    return levels * (1.0 + 0.01 * torch.arange(heads, device="cuda", dtype=torch.float32))[:, None]


def _packed(users, heads, keys, gen, codebooks, ids, signs=True, outliers=False):
    """Packed rows of ``users`` x ``heads`` x ``keys`` fresh keys (or values), a few users at a time."""
    nib = torch.empty(users, heads, keys, 64, dtype=torch.uint8, device="cuda")
    qjl = torch.empty(users, heads, keys, 8, dtype=torch.uint8, device="cuda") if signs else None
    norms = torch.empty(users, heads, keys, device="cuda") if signs else None
    chunk = max(1, min(users, (1 << 27) // (heads * keys * HEAD_DIM)))
    for u in range(0, users, chunk):
        n = min(chunk, users - u)
        rotate_quantize_append(_rows((n, heads, keys, HEAD_DIM), gen, torch.bfloat16, outliers), nib[u:u + n],
                               qjl[u:u + n] if signs else None, norms[u:u + n] if signs else None, 0, codebooks, ids[u:u + n])
    return nib, qjl, norms


def _lengths(case, gen):
    low = max(1, int(case["ragged"] * case["keys"]))
    return torch.randint(low, case["keys"] + 1, (case["users"],), generator=gen, device="cuda", dtype=torch.int32)


def _mean_keys(case):
    if not case["ragged"]:
        return float(case["keys"])
    return (max(1, int(case["ragged"] * case["keys"])) + case["keys"]) / 2.0


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "calibrate":
        # rotated rows of each head, heads of slightly different spread
        return dict(case=case, groups=[torch.randn(case["samples"], generator=gen, device="cuda") * (1.0 + 0.05 * g)
                                       for g in range(case["groups"])])
    users, heads = case["users"], case["kv_heads"]
    ids = torch.arange(users, dtype=torch.int32, device="cuda")
    if kind == "append":
        T, dtype = case["new_tokens"], DTYPES[case["dtype"]]
        shape, room = (users, heads, T, HEAD_DIM), T + 8
        k, v = _rows(shape, gen, dtype, heavy=True), _rows(shape, gen, dtype, heavy=True)
        bytes_ = lambda n: torch.zeros(users, heads, room, n, dtype=torch.uint8, device="cuda")  # noqa: E731
        floats = lambda: torch.zeros(users, heads, room, device="cuda")  # noqa: E731
        signs = case["v_signs"]
        return dict(case=case, k=k, v=v, ids=ids, codebooks=_codebooks(case["per_head"], heads, 1.41),
                    k_cache=(bytes_(64), bytes_(8), floats()),
                    v_cache=(bytes_(64), bytes_(8) if signs else None, floats() if signs else None))
    if kind == "bake":
        return dict(case=case, x=_rows((users, heads, case["keys"], HEAD_DIM), gen, DTYPES[case["dtype"]]), codebooks=_codebooks(True, heads))
    if kind == "dequantize":
        codebooks = _codebooks(True, heads)
        return dict(case=case, packed=_packed(users, heads, case["keys"], gen, codebooks, ids), codebooks=codebooks, ids=ids)

    q_heads, keys, dtype = case["q_heads"], case["keys"], DTYPES[case["dtype"]]
    if kind == "step":
        T = case["new_tokens"]
        codebooks = _codebooks(True, heads)
        cache = QuantizedKVCache(users, heads, keys + T, codebooks, "cuda", user_ids=ids)
        cache.append(_rows((users, heads, keys, HEAD_DIM), gen, dtype), _rows((users, heads, keys, HEAD_DIM), gen, dtype))
        return dict(case=case, cache=cache, lens=_lengths(case, gen).to(torch.int64),
                    k=_rows((users, heads, T, HEAD_DIM), gen, dtype), v=_rows((users, heads, T, HEAD_DIM), gen, dtype),
                    q=torch.randn(users, q_heads, T, HEAD_DIM, generator=gen, device="cuda", dtype=dtype))
    per_head, outliers = case.get("per_head", False), case.get("outliers", False)
    codebooks = _codebooks(per_head, heads, 1.72 if outliers else 1.0)
    lens = _lengths(case, gen) if case["ragged"] else None
    k_nib, k_qjl, k_norms = _packed(users, heads, keys, gen, codebooks, ids, outliers=outliers)
    if kind == "host":
        v_nib = _packed(users, heads, keys, gen, codebooks, ids, signs=False)[0]
        pair_v_rows(v_nib, 0, keys if lens is None else lens.to(torch.int64))
        step = HostDecodeStep(k_nib, k_qjl, k_norms, v_nib, codebooks, n_heads=q_heads, batch=users, q_dtype=dtype, user_id=ids,
                              seq_lens=lens, v_paired=True)
        step.q_host.copy_(torch.randn(users, q_heads, 1, HEAD_DIM, generator=gen, device="cuda", dtype=dtype))
        return dict(case=case, step=step)
    options = dict(user_id=ids)
    if case["lora_rank"]:
        # the benchmark's serving loop keeps one adapter pool and lets V share K's codes
        rank, v_nib = case["lora_rank"], k_nib
        options.update(x=torch.randn(users, 1, 128, generator=gen, device="cuda"),
                       lora_a=torch.randn(16, rank, 128, generator=gen, device="cuda") * 0.25,
                       lora_b=torch.randn(16, q_heads * HEAD_DIM, rank, generator=gen, device="cuda") * 0.05,
                       lora_indices=torch.randint(-1, 16, (users,), generator=gen, device="cuda", dtype=torch.int32),
                       lora_alpha=1.0 / rank)
    else:
        v_nib = _packed(users, heads, keys, gen, codebooks, ids, signs=False, outliers=outliers)[0]
    if case["pair"]:
        pair_v_rows(v_nib, 0, keys if lens is None else lens.to(torch.int64))
        options["v_paired"] = True
    if lens is not None:
        options["seq_lens"] = lens
    if case["rotated"]:
        options.update(rotate_q=True, unrotate_out=True)
    q = torch.randn(users, q_heads, case["tokens"], HEAD_DIM, generator=gen, device="cuda", dtype=dtype)
    return dict(case=case, args=(q, k_nib, k_qjl, k_norms, v_nib, codebooks), options=options)


def run(state):
    kind = state["case"]["kind"]
    if kind == "decode":
        return omni_attn(*state["args"], **state["options"])
    if kind == "step":
        cache = state["cache"]
        cache.lens.copy_(state["lens"])          # back to the end of the prompt, as for another continuation of it
        cache.append(state["k"], state["v"])
        out = cache.attend(state["q"], rotate_q=True, unrotate_out=True)
        return out, cache.lens, cache.k_nib, cache.k_qjl, cache.k_norms, cache.v_nib, cache.v_qjl, cache.v_norms
    if kind == "append":
        rotate_quantize_append(state["k"], *state["k_cache"], 3, state["codebooks"], state["ids"])
        rotate_quantize_append(state["v"], *state["v_cache"], 3, state["codebooks"], state["ids"])
        return [t for t in state["k_cache"] + state["v_cache"] if t is not None]
    if kind == "bake":
        return quantize_heads(rotate_queries(state["x"]), state["codebooks"], user_id=7)
    if kind == "dequantize":
        return dequantize_heads(*state["packed"], state["codebooks"], state["ids"], state["case"]["with_qjl"])
    if kind == "calibrate":
        return calibrate_per_group(state["groups"])
    return state["step"].step()


def work(case):
    kind = case["kind"]
    if kind == "calibrate":
        n = case["groups"] * case["samples"]
        return {"bytes": 4 * n + 64 * case["groups"], "flops": 32 * n}
    users, heads = case["users"], case["kv_heads"]
    wht = 7 * HEAD_DIM + HEAD_DIM
    encode = 4 * HEAD_DIM + 2 * HEAD_DIM * 64
    if kind == "append":
        rows, esz = users * heads * case["new_tokens"], DTYPE_BYTES[case["dtype"]]
        return {"bytes": rows * (2 * HEAD_DIM * esz + ROW_BYTES + (ROW_BYTES if case["v_signs"] else 64)),
                "flops": rows * (2 * wht + encode + (encode if case["v_signs"] else 4 * HEAD_DIM))}
    if kind == "bake":
        rows = users * heads * case["keys"]
        return {"bytes": rows * (HEAD_DIM * DTYPE_BYTES[case["dtype"]] + ROW_BYTES), "flops": rows * (wht + encode)}
    if kind == "dequantize":
        rows, signs = users * heads * case["keys"], case["with_qjl"]
        return {"bytes": rows * ((ROW_BYTES if signs else 64) + 4 * HEAD_DIM), "flops": rows * (HEAD_DIM * (66 if signs else 1))}
    q_heads, tokens = case["q_heads"], case.get("tokens", 1)
    keys = _mean_keys(case)
    extra_bytes = extra_flops = 0.0
    if kind == "step":
        tokens = case["new_tokens"]
        keys += tokens
        rows = users * heads * tokens
        extra_bytes = rows * 2 * (HEAD_DIM * DTYPE_BYTES[case["dtype"]] + ROW_BYTES)
        extra_flops = rows * 2 * (wht + encode)
    key_bytes = KEY_BYTES
    if case.get("lora_rank"):
        key_bytes = ROW_BYTES
        extra_bytes = 4 * case["lora_rank"] * min(16, users) * (128 + q_heads * HEAD_DIM) + users * 516
        extra_flops = 2.0 * users * case["lora_rank"] * (128 + q_heads * HEAD_DIM)
    rows = users * q_heads * tokens
    return {"bytes": users * heads * keys * key_bytes + rows * HEAD_DIM * (DTYPE_BYTES[case["dtype"]] + 4) + extra_bytes,
            "flops": rows * keys * (4 * HEAD_DIM + 2 * 64) + extra_flops}


def tolerance(case):
    kind = case["kind"]
    if kind in ("append", "bake"):
        return {"rel": 2e-6, "max": 2e-5, "differ": 0.0}            # codes and sign bits as they are, norms are fp32 sums
    if kind == "dequantize":
        return {"rel": 1e-6, "max": 1e-5}
    if kind == "calibrate":
        return {"rel": 1e-5, "max": 1e-4}
    if case["keys"] < 128 and users_rows(case) < 1024 and kind != "step":
        return {"rel": 2e-6, "max": 2e-5}                            # small calls: fp32 throughout (seen: 4e-7, 4e-6)
    return {"rel": 2.4e-3, "max": 3e-2, "differ": 0.0}               # fp16 tensor-core operands (seen: 6e-4, 7.5e-3)


def users_rows(case):
    return case["users"] * case["q_heads"] * case.get("tokens", 1)

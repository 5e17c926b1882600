"""The performance cases of the packed KV-cache path: what a serving program has it do.

A case is one of these kinds of work, at given sizes:

  decode   one decode-attention call over paged packed K/V (`packed_decode_attention`)
  session  one layer of a serving loop's decode step: append + attention (`DecodeSession.layer`)
  forward  the attention work of one batched decode forward through the Transformers interface:
           a `PagedPackedCache`, then append + attention in every layer
  prompt   the same for one prefill chunk of one request
  prefill  one causal attention call of a batch's query chunks (`packed_prefill_attention`)
  dequant  reconstruction of packed rows (`dequantize_rows`)
  legacy   the contiguous cache: a prompt, then one token (`TQPackedLayer.update`)

K and V are N(0, 1) with 2 % of the channels scaled by 8 (activation outliers), queries
N(0, 1) / sqrt(head_dim); pages are filled with the codes of such vectors.
"""
from __future__ import annotations

import math
import random

import torch

from winnow_b200 import packed_attention as pa
from winnow_b200 import packed_backend as pb
from winnow_b200.cache import TQPackedLayer, _get_quantizer, dequantize_rows
from winnow_b200.engine_step import DecodeSession
from winnow_b200.packed_attention_cuda import (decode_workspace, packed_decode_attention,
                                               packed_prefill_attention)
from winnow_b200.page_pool import PagePool

DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}


def _case(kind, name=None, **kw):
    c = {"name": name, "kind": kind} if name else {"kind": kind}
    c.update(kw)
    return c


def _attn(kind, name=None, *, batch, q_heads, kv_heads, lo, hi, page=16, bits_k=4, bits_v=4,
          dtype="fp16", head_dim=128, **kw):
    """Contexts are log-uniform in [lo, hi] (all equal when lo == hi)."""
    return _case(kind, name, batch=batch, q_heads=q_heads, kv_heads=kv_heads, head_dim=head_dim,
                 lo=lo, hi=hi, page=page, bits_k=bits_k, bits_v=bits_v, dtype=dtype, **kw)


def listed():
    return [
        # a single short chat on a small model: the smallest call, where latency counts
        _attn("decode", "decode_b1_1k", batch=1, q_heads=8, kv_heads=2, lo=1024, hi=1024, dtype="fp32"),
        # an 8B model's usual serving batch: the benchmark's default workload
        _attn("decode", "decode_b16_8k", batch=16, q_heads=32, kv_heads=8, lo=8192, hi=8192),
        # one very long document, one stream
        _attn("decode", "decode_b1_128k", batch=1, q_heads=64, kv_heads=8, lo=131072, hi=131072, page=64),
        # a full server with requests of all lengths, keys narrower than values
        _attn("decode", "decode_b128_ragged", batch=128, q_heads=32, kv_heads=8, lo=512, hi=32768,
              bits_v=6),
        # 8-bit codes, seven query heads to a kv head, short odd contexts: many small requests
        _attn("decode", "decode_b32_8bit", batch=32, q_heads=28, kv_heads=4, lo=37, hi=1973, page=32,
              bits_k=8, bits_v=8, dtype="bf16"),
        # a half-billion-parameter model: head_dim 64
        _attn("decode", "decode_b8_d64", batch=8, q_heads=14, kv_heads=2, lo=700, hi=5000, head_dim=64,
              dtype="bf16"),
        # one layer of a serving loop at 6 bits: fused append and attention
        _attn("session", "session_b32_16k_6bit", batch=32, q_heads=32, kv_heads=8, lo=16384, hi=16384,
              bits_k=6, bits_v=6, graph=False),
        # a decode forward as the engine issues it for a 7B model, eight layers of it
        _attn("forward", "forward_b8_layers8", batch=8, q_heads=28, kv_heads=4, lo=300, hi=4100,
              dtype="bf16", layers=8),
        # a 512-token chunk in the middle of a long prompt
        _attn("prompt", "prompt_512_of_4k", batch=1, q_heads=32, kv_heads=8, lo=3584, hi=3584,
              dtype="bf16", layers=2, new=512),
        # chunked prefill of a whole batch over long histories
        _attn("prefill", "prefill_b16_q64_8k", batch=16, q_heads=32, kv_heads=8, lo=8192, hi=8192, new=64),
        # reconstruction of a long history for stock attention
        _case("dequant", "dequant_1m_rows", batch=8, kv_heads=4, length=32768, max_length=32768,
              head_dim=128, bits=4, dtype="bf16"),
        # the contiguous cache: a prompt of a small batch, then the first generated token
        _case("legacy", "legacy_b4_2k", batch=4, kv_heads=8, length=1999, max_length=4096, head_dim=128,
              bits=4, dtype="fp16"),
    ]


# ---- drawn cases ---------------------------------------------------------------------------
MAX_BYTES = 1.0e9             # of cached codes and norms one pass reads
MAX_PREFILL_FLOPS = 1.3e11
WIDTHS = ((4, 4), (4, 4), (4, 6), (6, 6), (8, 8))
HEADS = ((8, 2), (16, 8), (28, 4), (32, 8), (64, 8))


def _log(rng: random.Random, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _token_bytes(c) -> int:
    """Bytes one cached token of one kv head occupies."""
    return c["head_dim"] * (c["bits_k"] + c["bits_v"]) // 8 + 4


def draw(rng: random.Random):
    kind = rng.choice(("decode", "decode", "decode", "session", "forward", "prompt", "prefill",
                       "dequant", "legacy"))
    if kind == "dequant":
        dtype = rng.choice(("fp16", "bf16", "bf16", "fp32"))
        batch, heads = _log(rng, 1, 16), rng.choice((2, 4, 8))
        length = min(_log(rng, 500, 32768), (1 << (18 if dtype == "fp32" else 20)) // (batch * heads))
        return _case(kind, batch=batch, kv_heads=heads, length=length,
                     max_length=length + rng.choice((0, 1, 777)), head_dim=rng.choice((64, 128, 128, 128)),
                     bits=rng.choice((4, 4, 6, 8)), dtype=dtype)
    if kind == "legacy":
        batch, heads = _log(rng, 1, 8), rng.choice((2, 4, 8))
        length = min(_log(rng, 100, 8192), (1 << 16) // (batch * heads))
        return _case(kind, batch=batch, kv_heads=heads, length=length, max_length=length + 1000,
                     head_dim=128, bits=rng.choice((4, 4, 6, 8)), dtype=rng.choice(("fp16", "bf16")))
    (bits_k, bits_v), (q_heads, kv_heads) = rng.choice(WIDTHS), rng.choice(HEADS)
    c = _attn(kind, batch=1, q_heads=q_heads, kv_heads=kv_heads, lo=1, hi=1, page=rng.choice((16, 16, 32, 64)),
              bits_k=bits_k, bits_v=bits_v, dtype=rng.choice(("fp16", "bf16", "bf16")))
    if kind == "decode" and rng.random() < 0.2:                 # small models: head_dim 64
        c.update(head_dim=64, q_heads=14, kv_heads=2)
    if kind == "prompt":
        c.update(layers=2, new=_log(rng, 33, 1024), lo=_log(rng, 1, 16384))
        c["hi"] = c["lo"]
        return c
    if kind == "prefill":
        c.update(batch=_log(rng, 1, 32), new=_log(rng, 2, 256))
        room = MAX_PREFILL_FLOPS / (4.0 * c["batch"] * c["new"] * c["q_heads"] * c["head_dim"])
        c["hi"] = max(c["new"] + 1, min(_log(rng, 300, 32768), int(room)))
        c["lo"] = rng.choice((c["hi"], max(c["new"], c["hi"] // 4)))
        return c
    c["batch"] = _log(rng, 1, 64 if kind == "forward" else 128)
    layers = 1
    if kind == "forward":
        layers = c["layers"] = 4
    if kind == "session":
        c["graph"] = rng.random() < 0.5
    room = MAX_BYTES / (c["batch"] * c["kv_heads"] * layers * _token_bytes(c))
    c["hi"] = max(16, min(_log(rng, 100, 131072 if c["batch"] == 1 else 32768), int(room)))
    c["lo"] = rng.choice((c["hi"], max(1, c["hi"] // 8), max(1, c["hi"] // 64)))
    return c


# ---- inputs --------------------------------------------------------------------------------
def _lengths(c, seed: int) -> list[int]:
    """Tokens each sequence holds when the pass has run, whatever the kind."""
    rng = random.Random(seed * 7919 + 13)
    lens = [_log(rng, c["lo"], c["hi"]) for _ in range(c["batch"])]
    if c["kind"] == "prefill":
        lens = [max(n, c["new"]) for n in lens]
    return lens


def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _vectors(g, *shape, dtype=torch.float32):
    """N(0, 1) with the last channels of each vector as outliers."""
    x = torch.randn(*shape, device="cuda", generator=g)
    x[..., -max(1, round(0.02 * shape[-1])):] *= 8.0
    return x.to(dtype)


def _fill_pages(pool: PagePool, g, kq, vq, head_dim: int) -> None:
    """Every slot of every page holds the codes of a vector of its own."""
    for pages, norms, tq in ((pool.k_pages, pool.k_norms, kq), (pool.v_pages, pool.v_norms, vq)):
        rows, flat = pages.view(-1, pages.shape[-1]), norms.view(-1)
        for at in range(0, rows.shape[0], 1 << 20):
            x = _vectors(g, min(1 << 20, rows.shape[0] - at), head_dim)
            codes, n = tq.quantize(x, packed=True)
            rows[at:at + x.shape[0]] = codes
            flat[at:at + x.shape[0]] = n.half()


def _quantizers(c):
    return (_get_quantizer(c["bits_k"], c["head_dim"], "cuda", 42),
            _get_quantizer(c["bits_v"], c["head_dim"], "cuda", 43))


def _pool(c, longest: int, g):
    """Room for every sequence at the longest length the case allows."""
    kq, vq = _quantizers(c)
    D, S = c["head_dim"], c["page"]
    pool = PagePool(num_layers=c.get("layers", 1), num_pages=c["batch"] * -(-longest // S),
                    num_kv_heads=c["kv_heads"], page_size=S, nb_k=D * c["bits_k"] // 8,
                    nb_v=D * c["bits_v"] // 8, device="cuda")
    _fill_pages(pool, g, kq, vq, D)
    return pool, kq, vq


def _reserve(pool: PagePool, lens) -> list[str]:
    """Requests that grew side by side, as in a running server: their pages alternate."""
    owners = [f"request{b}" for b in range(len(lens))]
    done, step = 0, 16 * pool.page_size
    while done < max(lens):
        done += step
        pool.ensure_many(owners, [min(done, n) for n in lens])
    return owners


def _queries(g, c, new: int):
    q = torch.randn(c["batch"], c["q_heads"], new, c["head_dim"], device="cuda", generator=g)
    return (q / math.sqrt(c["head_dim"])).to(DTYPES[c["dtype"]])


def _prepare_operator(c, seed: int):
    g, lens = _generator(seed), _lengths(c, seed)
    pool, kq, vq = _pool(c, max(c["hi"], c.get("new", 1)), g)
    S = c["page"]
    order = torch.randperm(pool.num_pages, device="cuda", generator=g).to(torch.int32)
    need = [-(-n // S) for n in lens]
    table, at = torch.full((c["batch"], max(need)), -1, dtype=torch.int32, device="cuda"), 0
    for b, n in enumerate(need):
        table[b, :n] = order[at:at + n]
        at += n
    kv = pa.PackedKV(pool.k_pages[0], pool.k_norms[0], pool.v_pages[0], pool.v_norms[0], table,
                     torch.tensor(lens, dtype=torch.int32, device="cuda"), pa.Quantizer.from_tq(kq),
                     pa.Quantizer.from_tq(vq), c["head_dim"])
    q = _queries(g, c, c.get("new", 1))
    state = {"kind": c["kind"], "q": q, "kv": kv, "scale": c["head_dim"] ** -0.5}
    if c["kind"] == "decode":
        state["out"] = torch.empty_like(q)
        state["workspace"] = decode_workspace(c["batch"], c["q_heads"], c["kv_heads"], c["head_dim"],
                                              table.shape[1], S, 0, q.device)
    return state


def _prepare_session(c, seed: int):
    g, lens = _generator(seed), _lengths(c, seed)
    pool, kq, vq = _pool(c, c["hi"], g)
    owners = _reserve(pool, lens)
    dtype, B, D = DTYPES[c["dtype"]], c["batch"], c["head_dim"]
    s = DecodeSession(pool, owners, [n - 1 for n in lens], k_quant=kq, v_quant=vq, head_dim=D,
                      q_heads=c["q_heads"], dtype=dtype, max_tokens=max(lens))
    s.begin_step()
    if c["graph"]:
        s.capture()
    return {"kind": "session", "session": s, "pool": pool, "q": _queries(g, c, 1),
            "k": _vectors(g, B, c["kv_heads"], 1, D, dtype=dtype),
            "v": _vectors(g, B, c["kv_heads"], 1, D, dtype=dtype)}


def _prepare_forward(c, seed: int):
    """`forward`: one new token per sequence; `prompt`: c["new"] tokens after lo stored ones."""
    new = c.get("new", 1)
    g = _generator(seed)
    lens = [c["lo"] + new] if c["kind"] == "prompt" else _lengths(c, seed)
    pool, kq, vq = _pool(c, max(lens) if c["kind"] == "prompt" else c["hi"], g)
    owners = _reserve(pool, lens)
    dtype, B, D = DTYPES[c["dtype"]], c["batch"], c["head_dim"]
    layers = [(_queries(g, c, new), _vectors(g, B, c["kv_heads"], new, D, dtype=dtype),
               _vectors(g, B, c["kv_heads"], new, D, dtype=dtype)) for _ in range(c["layers"])]
    return {"kind": c["kind"], "pool": pool, "owners": owners, "lengths": [n - new for n in lens],
            "layers": layers, "kq": kq, "vq": vq, "head_dim": D}


def _prepare_rows(c, seed: int):
    g = _generator(seed)
    B, H, L, D = c["batch"], c["kv_heads"], c["length"], c["head_dim"]
    dtype = DTYPES[c["dtype"]]
    if c["kind"] == "legacy":
        layer = TQPackedLayer(D, c["bits"], "cuda", c["max_length"])
        prompt = [_vectors(g, B, H, L, D, dtype=dtype) for _ in range(2)]
        token = [_vectors(g, B, H, 1, D, dtype=dtype) for _ in range(2)]
        return {"kind": "legacy", "layer": layer, "prompt": prompt, "token": token}
    tq = _get_quantizer(c["bits"], D, "cuda", 42)
    codes = torch.empty(B, H, c["max_length"], D * c["bits"] // 8, dtype=torch.uint8, device="cuda")
    norms = torch.empty(B, H, c["max_length"], dtype=torch.float16, device="cuda")
    for b in range(B):
        rows, n = tq.quantize(_vectors(g, H, c["max_length"], D), packed=True)
        codes[b], norms[b] = rows, n.half()
    return {"kind": "dequant", "codes": codes[:, :, :L], "norms": norms[:, :, :L], "tq": tq,
            "out": torch.empty(B, H, L, D, dtype=dtype, device="cuda")}


def prepare(case, seed):
    c = dict(case)
    if c["kind"] in ("decode", "prefill"):
        return _prepare_operator(c, seed)
    if c["kind"] == "session":
        return _prepare_session(c, seed)
    if c["kind"] in ("forward", "prompt"):
        return _prepare_forward(c, seed)
    return _prepare_rows(c, seed)


# ---- one pass ------------------------------------------------------------------------------
def _pages(pool: PagePool):
    return [pool.k_pages, pool.k_norms, pool.v_pages, pool.v_norms]


def run(s):
    kind = s["kind"]
    if kind == "decode":
        return packed_decode_attention(s["q"], s["kv"], s["scale"], check_page_ids=False,
                                       out=s["out"], workspace=s["workspace"])
    if kind == "prefill":
        return packed_prefill_attention(s["q"], s["kv"], s["scale"], check_page_ids=False)
    if kind == "session":
        return [s["session"].layer(0, s["k"], s["v"], s["q"])] + _pages(s["pool"])
    if kind in ("forward", "prompt"):
        cache = pb.PagedPackedCache(s["pool"], s["owners"], s["lengths"], k_quant=s["kq"],
                                    v_quant=s["vq"], head_dim=s["head_dim"])
        outs = []
        for i, (q, k, v) in enumerate(s["layers"]):
            key, value = cache.update(k, v, i)
            outs.append(pb.winnow_packed_attention(None, q, key, value, None)[0])
        return outs + _pages(s["pool"])
    if kind == "legacy":
        s["layer"].reset()
        s["layer"].update(*s["prompt"])
        return s["layer"].update(*s["token"])
    tq = s["tq"]
    return dequantize_rows(s["codes"], s["norms"], tq.centroids, tq.Pi, tq.bit_width, tq.head_dim,
                           out=s["out"])


# ---- what a pass cannot do without ---------------------------------------------------------
def work(case):
    c = dict(case)
    D, el = c["head_dim"], 4 if c["dtype"] == "fp32" else 2
    if c["kind"] in ("dequant", "legacy"):
        rows, nb = c["batch"] * c["kv_heads"] * c["length"], D * c["bits"] // 8
        if c["kind"] == "dequant":
            return {"bytes": rows * (nb + 2 + D * el), "flops": 2.0 * rows * D * D}
        # K and V: read the prompt, write its codes, reconstruct it twice (prompt, then token)
        return {"bytes": 2 * rows * (D * el + nb + 2 + 2 * (nb + 2 + D * el)),
                "flops": 2 * 3 * 2.0 * rows * D * D}
    new, layers = c.get("new", 1), c.get("layers", 1)
    if c["kind"] == "prompt":
        tokens = c["lo"] + new
    else:                     # mean of the log-uniform law
        lo, hi = c["lo"], c["hi"]
        tokens = lo if lo == hi else (hi - lo) / math.log(hi / lo)
        tokens = max(tokens, new)
    queries, heads = c["batch"] * new * c["q_heads"], c["kv_heads"]
    nbytes = c["batch"] * tokens * heads * _token_bytes(c) + 2 * queries * D * el \
        + 4 * c["batch"] * -(-int(tokens) // c["page"])
    flops = 4.0 * queries * D * (tokens - (new - 1) / 2) + 4.0 * queries * D * D
    if c["kind"] in ("session", "forward", "prompt"):
        vectors = 2 * c["batch"] * heads * new
        nbytes += vectors * D * el + vectors * _token_bytes(c) // 2
        flops += 2.0 * vectors * D * D
    return {"bytes": layers * nbytes, "flops": layers * flops}


def tolerance(case):
    """Operands of the attention contractions are 16-bit floats (11-bit significands) and sums
    are fp32: two correct implementations of it stay within 1e-3, and outputs rounded to bf16
    within 5e-3.  Packed codes are whole numbers and the same in every implementation.  fp32
    reconstruction is fp32 arithmetic throughout."""
    if case["dtype"] == "bf16":
        return {"rel": 5e-3}
    if case["kind"] == "dequant" and case["dtype"] == "fp32":
        return {"rel": 1e-5}
    return {"rel": 1e-3}

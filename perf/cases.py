"""Performance cases of the compressed KV cache: what a serving program has this package do.

A case is one pass through the public entry points at one shape:

  step          a decode step of a serving engine on the paged pool: the new token of every
                sequence is stored, then attention runs over the whole context
  store         prefill: the K and V of a prompt are encoded into the paged pool
  continuation  causal attention of several new tokens per sequence over the cache (chunked
                prefill, speculative verification)
  flash         decode attention over contiguous compressed K / V (the Hugging Face cache format)
  quantizer     TurboQuantMSE: encode a tensor of head vectors, decode it again
  slot_store    prefill into the vLLM-v1 slot format
  slot_decode   a decode step's attention over the vLLM-v1 slot format

Inputs are synthetic: K and V are normal with 1 % of the channels ten times larger (the outlier
channels of real keys), page tables are shuffled, queries are normal.
"""
import math

import torch

from fused_turboquant_b200 import PagedKVPool, TurboQuantMSE
from fused_turboquant_b200 import kernels, tq_v1

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
PAGE = 16
MAX_STEP_BYTES = 250e6       # drawn cases stay below the listed ones' largest
MAX_EXACT_BYTES = 40e6       # ... where the arithmetic is fp32 throughout
MAX_STORE_VECTORS = 1 << 18


def listed():
    return [
        # one chat on a local machine: a short context, every microsecond of launch shows
        dict(name="step_single", kind="step", batch=1, ctx=900, ragged=False, hq=32, hkv=8, d=128,
             kb=4, vb=4, layers=1, dtype="bf16"),
        # a small model served in batch, all layers in one call
        dict(name="step_small_model", kind="step", batch=32, ctx=4096, ragged=False, hq=14, hkv=2,
             d=64, kb=3, vb=3, layers=24, dtype="bf16"),
        # one layer of the headline serving batch
        dict(name="step_serving", kind="step", batch=64, ctx=8192, ragged=False, hq=32, hkv=8,
             d=128, kb=4, vb=4, layers=1, dtype="bf16"),
        # one layer of a long-context batch, GQA group 8
        dict(name="step_long", kind="step", batch=4, ctx=131072, ragged=False, hq=64, hkv=8, d=128,
             kb=3, vb=3, layers=1, dtype="bf16"),
        # a mixed batch: contexts log-uniform up to 32k, 2-bit values, head_dim 256
        dict(name="step_ragged", kind="step", batch=256, ctx=32768, ragged=True, hq=16, hkv=8,
             d=256, kb=4, vb=2, layers=1, dtype="bf16"),
        # a prompt batch encoded into the pool
        dict(name="store_prefill", kind="store", tokens=32768, hkv=8, d=128, kb=4, vb=4,
             dtype="bf16"),
        # a chunk of new tokens against its cached context
        dict(name="continuation_chunk", kind="continuation", batch=4, q_len=64, ctx=4096, hq=32,
             hkv=8, d=128, kb=4, vb=4, dtype="bf16"),
        # decode step of the Hugging Face cache, which hands over fp32 queries already rotated
        dict(name="flash_fp32", kind="flash", batch=4, ctx=4001, hq=32, hkv=8, d=128, kb=4, vb=4,
             dtype="fp32"),
        # the quantizer on a layer's keys
        dict(name="quantizer_roundtrip", kind="quantizer", vectors=8 * 4097, d=128, kb=4,
             dtype="fp16"),
        # a prompt batch into the slot format, values rotated as the small-model preset has it
        dict(name="slot_store_prefill", kind="slot_store", tokens=16384, hkv=8, d=128, kb=4, vb=4,
             v_rotate=True, dtype="bf16"),
        # one layer of a serving batch in the slot format
        dict(name="slot_decode_serving", kind="slot_decode", batch=32, ctx=8192, ragged=False,
             hq=32, hkv=8, d=128, kb=4, vb=4, v_rotate=False, layers=1, dtype="bf16"),
        # the FP8-key preset of the slot format
        dict(name="slot_decode_fp8_keys", kind="slot_decode", batch=16, ctx=4096, ragged=False,
             hq=32, hkv=8, d=128, kb=8, vb=4, v_rotate=False, layers=1, dtype="bf16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "store", "continuation", "flash", "quantizer",
                       "slot_store", "slot_decode", "slot_decode"])
    d = rng.choice([64, 128, 128, 128, 256])
    hkv, group = rng.choice([1, 2, 4, 8]), rng.choice([1, 2, 4, 4, 7, 8])
    kb, vb = rng.choice([2, 3, 4, 4]), rng.choice([2, 3, 4, 4])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    if kind == "store":
        return dict(kind=kind, tokens=_log_int(rng, 16, MAX_STORE_VECTORS // hkv * 64 // d), hkv=hkv,
                    d=d, kb=kb, vb=vb, dtype=dtype)
    if kind == "quantizer":
        return dict(kind=kind, vectors=_log_int(rng, 8, MAX_STORE_VECTORS * 32 // d), d=d, kb=kb,
                    dtype=rng.choice(["fp16", "bf16", "fp32"]))
    if kind == "slot_store":
        return dict(kind=kind, tokens=_log_int(rng, 16, MAX_STORE_VECTORS // 2 // hkv * 64 // d),
                    hkv=hkv, d=d, kb=rng.choice([3, 4, 4, 8]), vb=rng.choice([3, 4, 4]),
                    v_rotate=rng.random() < 0.5, dtype=dtype)
    if kind == "slot_decode":
        kb, vb, d = rng.choice([3, 4, 4, 8]), rng.choice([3, 4, 4]), rng.choice([64, 128, 128])
    exact = kind == "flash" or kb == 8
    if kind == "flash":
        dtype = rng.choice(["fp32", "fp32", "bf16"])
    elif kind == "step" and rng.random() < 0.15:
        dtype, exact = "fp32", True
    batch = _log_int(rng, 1, 8 if kind == "continuation" else 128)
    q_len = _log_int(rng, 2, 128) if kind == "continuation" else 1
    cap = (MAX_EXACT_BYTES if exact else MAX_STEP_BYTES) / q_len
    per_token = batch * hkv * _token_bytes(kind, d, kb, vb)
    top = max(64, min(65536 if kind != "continuation" else 8192, int(cap / per_token)))
    ctx = _log_int(rng, 64, top)
    ctx = max(ctx, q_len)
    case = dict(kind=kind, batch=batch, ctx=ctx, hq=hkv * group, hkv=hkv, d=d, kb=kb, vb=vb,
                dtype=dtype)
    if kind == "continuation":
        case["q_len"] = q_len
    if kind in ("step", "slot_decode"):
        case["ragged"] = rng.random() < 0.4
        room = int(cap / (per_token * ctx))
        case["layers"] = rng.choice([1, max(1, min(24, room))])
    if kind == "slot_decode":
        case["v_rotate"] = rng.random() < 0.5
    return case


def _token_bytes(kind, d, kb, vb):
    """Bytes of one (token, KV head): codes and fp16 norms; the slot format has a scale and a zero
    point per value vector, and no norm behind FP8 keys."""
    if kind.startswith("slot"):
        return d * kb // 8 + (0 if kb == 8 else 2) + d * vb // 8 + 4
    return d * kb // 8 + 2 + d * vb // 8 + 2


def _lens(case):
    """Context lengths of the batch (host): equal, or log-uniform in [ctx / 256, ctx] with the
    longest at ctx (a fixed mix, so that a case is the same amount of work for every seed)."""
    if not case.get("ragged"):
        return [case["ctx"]] * case["batch"]
    g = torch.Generator("cpu").manual_seed(20250)
    lo = max(16, case["ctx"] // 256)
    u = torch.rand(case["batch"], generator=g).tolist()
    n = [int(math.exp(math.log(lo) + x * (math.log(case["ctx"]) - math.log(lo)))) for x in u]
    n[0] = case["ctx"]
    return n


def _vectors(shape, gen, dtype):
    """Head vectors [..., heads, d] with 1 % of the channels of each head ten times larger."""
    x = torch.randn(shape, device="cuda", generator=gen)
    wide = torch.rand(shape[-2:], device="cuda", generator=gen) < 0.01
    return torch.where(wide, x * 10.0, x).to(dtype)


def _pages(lens, gen, page=PAGE):
    """(block table [B, max_blocks], number of blocks, slots of all tokens, their offsets): the
    blocks of a batch in shuffled order."""
    per = [(n + page - 1) // page for n in lens]
    nb, width = sum(per), max(per)
    ids = torch.randperm(nb, device="cuda", generator=gen)
    table = torch.zeros(len(lens), width, dtype=torch.int32, device="cuda")
    first = torch.tensor([sum(per[:i]) for i in range(len(per))], device="cuda")
    count = torch.tensor(per, device="cuda")
    col = torch.arange(width, device="cuda")
    table[col[None, :] < count[:, None]] = ids.to(torch.int32)
    rows = torch.repeat_interleave(torch.arange(len(lens), device="cuda"), torch.tensor(lens, device="cuda"))
    start = torch.cumsum(torch.tensor([0] + lens[:-1], device="cuda"), 0)
    pos = torch.arange(sum(lens), device="cuda") - start[rows]
    return table, nb, ids[first[rows] + pos // page] * page + pos % page


def _last_slots(table, lens, page=PAGE):
    """Slot of the newest token of every sequence."""
    last = torch.tensor(lens, device="cuda") - 1
    blk = table.gather(1, (last // page)[:, None])[:, 0].long()
    return blk * page + last % page


def prepare(case, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    kind, d, dtype = case["kind"], case["d"], DTYPES[case["dtype"]]
    if kind == "quantizer":
        tq = TurboQuantMSE(d, bits=case["kb"], device="cuda")
        return dict(case=case, tq=tq, x=_vectors((case["vectors"], 1, d), gen, dtype)[:, 0])
    hkv, kb, vb = case["hkv"], case["kb"], case["vb"]
    if kind in ("store", "slot_store"):
        n = case["tokens"]
        _, nb, slots = _pages([n], gen)
        s = dict(case=case, key=_vectors((n, hkv, d), gen, dtype),
                 value=_vectors((n, hkv, d), gen, dtype), slots=slots)
        if kind == "store":
            s["pool"] = PagedKVPool(nb, hkv, d, kb, vb, device="cuda")
        else:
            s["cfg"], s["centroids"], s["midpoints"] = _slot_config(case)
            s["cache"] = torch.zeros((nb, PAGE, hkv, s["cfg"].slot_size_aligned),
                                     dtype=torch.uint8, device="cuda")
        return s
    lens, hq, B, layers = _lens(case), case["hq"], case["batch"], case.get("layers", 1)
    if kind == "flash":
        tk, tv = TurboQuantMSE(d, bits=kb, device="cuda"), TurboQuantMSE(d, bits=vb, device="cuda")
        k = tk.encode(_vectors((B, case["ctx"], hkv, d), gen, torch.bfloat16).transpose(1, 2).contiguous())
        v = tv.encode(_vectors((B, case["ctx"], hkv, d), gen, torch.bfloat16).transpose(1, 2).contiguous())
        q = torch.randn(B, hq, 1, d, device="cuda", generator=gen)
        q = tk.rotation(q) if dtype is torch.float32 else q.to(dtype)
        return dict(case=case, tk=tk, tv=tv, k=k, v=v, q=q)
    table, nb, slots = _pages(lens, gen)
    s = dict(case=case, table=table, lens=torch.tensor(lens, dtype=torch.int32, device="cuda"),
             top=max(lens))
    lead = (layers,) if layers > 1 else ()
    if kind == "slot_decode":
        cfg, s["centroids"], mids = _slot_config(case)
        s["cfg"] = cfg
        s["cache"] = torch.zeros(lead + (nb, PAGE, hkv, cfg.slot_size_aligned), dtype=torch.uint8,
                                 device="cuda")
        for layer in range(layers):
            cache = s["cache"][layer] if lead else s["cache"]
            for at in range(0, sum(lens), 1 << 17):
                part = slots[at:at + (1 << 17)]
                tq_v1.launch_store(_vectors((len(part), hkv, d), gen, torch.bfloat16),
                                   _vectors((len(part), hkv, d), gen, torch.bfloat16), cache, part,
                                   mids, cfg, v_rotate=case["v_rotate"])
        s["q"] = torch.randn(lead + (B, hq, d), device="cuda", generator=gen).to(dtype)
        # buffers that the engine keeps per layer
        s["splits"] = 8
        s["mid"] = torch.empty(layers * B, hq, 8, d + 1, dtype=torch.float32, device="cuda")
        s["out"] = torch.empty(lead + (B, hq, d), dtype=dtype, device="cuda")
        return s
    pool = s["pool"] = PagedKVPool(nb, hkv, d, kb, vb, n_layers=layers, device="cuda")
    for layer in range(layers):
        for at in range(0, sum(lens), 1 << 17):
            part = slots[at:at + (1 << 17)]
            pool.store(_vectors((len(part), hkv, d), gen, torch.bfloat16),
                       _vectors((len(part), hkv, d), gen, torch.bfloat16), part, layer=layer)
    if kind == "continuation":
        s["q"] = torch.randn(B, case["q_len"], hq, d, device="cuda", generator=gen).to(dtype)
        return s
    s["layer"] = None if lead else 0
    s["q"] = torch.randn(lead + (B, hq, d), device="cuda", generator=gen).to(dtype)
    s["key"] = _vectors(lead + (B, hkv, d), gen, dtype)
    s["value"] = _vectors(lead + (B, hkv, d), gen, dtype)
    s["new"] = _last_slots(table, lens)
    return s


def _slot_config(case):
    cfg = tq_v1.TurboQuantSlotConfig(case["d"], case["kb"], case["vb"], norm_correction=True)
    tq = TurboQuantMSE(case["d"], bits=case["kb"] if case["kb"] < 8 else case["vb"], device="cuda")
    cent, mids = tq_v1.midpoints_of(tq.quantizer.levels)
    return cfg, cent, mids


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "step":
        pool = s["pool"]
        pool.store(s["key"], s["value"], s["new"], layer=s["layer"])
        out = pool.decode_attention(s["q"], s["table"], s["lens"], s["top"], layer=s["layer"])
        return out, pool.pool
    if kind == "store":
        s["pool"].store(s["key"], s["value"], s["slots"], layer=0)
        return s["pool"].pool
    if kind == "continuation":
        return s["pool"].continuation_attention(s["q"], s["table"], s["lens"], s["top"])
    if kind == "flash":
        tk, tv, q = s["tk"], s["tv"], s["q"]
        return kernels.flash_decode_compressed(
            q, s["k"].indices, s["k"].norms, s["v"].indices, s["v"].norms, tk.quantizer.levels,
            tv.quantizer.levels, tk.rotation.signs, case["d"] ** -0.5, case["kb"], case["vb"],
            q_is_rotated=q.dtype is torch.float32, out_dtype=q.dtype)
    if kind == "quantizer":
        ct = s["tq"].encode(s["x"])
        return ct.indices, ct.norms, s["tq"].decode(ct)
    if kind == "slot_store":
        tq_v1.launch_store(s["key"], s["value"], s["cache"], s["slots"], s["midpoints"], s["cfg"],
                           v_rotate=case["v_rotate"])
        return s["cache"]
    return tq_v1.decode_attention(s["q"], s["cache"], s["table"], s["lens"], s["centroids"],
                                  s["cfg"], case["d"] ** -0.5, num_kv_splits=s["splits"],
                                  v_rotate=case["v_rotate"], mid_o=s["mid"], output=s["out"])


def work(case):
    kind, d, es = case["kind"], case["d"], DTYPES[case["dtype"]].itemsize
    if kind == "quantizer":
        # read the vectors, write codes and norms, write the fp32 vectors; two butterflies each
        n = case["vectors"]
        return dict(bytes=n * (d * es + d * case["kb"] // 8 + 2 + 4 * d),
                    flops=n * d * (2 * math.log2(d) + 6))
    tok = _token_bytes(kind, d, case["kb"], case["vb"])
    if kind in ("store", "slot_store"):
        n = case["tokens"] * case["hkv"]
        return dict(bytes=n * (2 * d * es + tok) + 8 * case["tokens"],
                    flops=2 * n * d * (math.log2(d) + 4))
    lens, layers, q_len = _lens(case), case.get("layers", 1), case.get("q_len", 1)
    out_es = es
    kv = layers * sum(lens) * case["hkv"] * tok + 4 * sum((n + 15) // 16 for n in lens)
    rows = layers * case["batch"] * q_len * case["hq"]
    new = 2 * layers * case["batch"] * case["hkv"] * d * es if kind == "step" else 0
    attended = sum(q_len * n - q_len * (q_len - 1) // 2 for n in lens)
    return dict(bytes=kv + rows * d * (es + out_es) + new,
                flops=4.0 * layers * attended * case["hq"] * d)


def tolerance(case):
    kind = case["kind"]
    if kind in ("store", "slot_store"):
        return "exact"                      # codes, norms, scales: bytes
    if kind == "quantizer":
        return dict(rel=1e-5)               # codes the same, fp32 sums
    if case["dtype"] == "fp32":
        return dict(rel=2e-5)               # fp32 softmax and sums over the context
    # queries, weights and centroids are 16-bit operands, the result is rounded to 16 bits
    return dict(rel=1e-2 if case["dtype"] == "bf16" else 4e-3)

"""The work that programs have this library do, as cases that can be timed and compared between two builds of it.

A case is a plain dict; `path` says which sequence of public calls it makes:

  train    one attention training step: forward with log-sum-exp, Delta pre-pass, backward (`flash_attention`)
  forward  attention forward alone, as an inference or scoring program calls it
  step     one token of one sequence through one layer: RoPE, KV write, decode attention, called from the host
  token    one token through the attention half of a stack of layers (qkv projection + RoPE + KV write in one call, decode
           attention, output projection), captured once in a CUDA graph and replayed per token
  batch    one token for each of many sequences over paged caches: a continuous-batching server's step of one layer
  long     decode attention alone over a few very long sequences, each with a contiguous cache
  prefill  a prompt's chunk: RoPE, KV write, causal attention over the cache
  layer    the same chunk with the projections either side of it

`listed()` gives the cases, `draw(rng)` more of the same ranges, `prepare` what a program holds before the call, `run` one
pass, `work` the bytes and operations a pass cannot do without, `tolerance` how far two right results may lie apart.
"""
import math

import torch

from mx230_b200 import _lib
from mx230_b200 import flash_attention as fa
from mx230_b200 import llm_attention as la
from mx230_b200.common import Handle

D = 64
BLOCK = la.KV_BLOCK
THETA = 1e6

_handle = None


def handle():
    """The program's handle: one per device, kept for the life of the process."""
    global _handle
    if _handle is None:
        _handle = Handle(torch.cuda.current_device(), 64 << 20)
    return _handle


def listed():
    return [
        # Training at the size of the benchmark's headline: 4 x 12 heads of 4096 tokens, the staged operands reused between
        # forward and backward as that benchmark does.
        {"name": "train 48x4096 causal", "path": "train", "heads": 48, "n": 4096, "causal": True, "bf16": False, "reuse": True},
        # A small model's training step with a ragged sequence length and every option at its default.
        {"name": "train 12x1000 causal", "path": "train", "heads": 12, "n": 1000, "causal": True, "bf16": False, "reuse": False},
        # An encoder's training step (no mask) whose activations are kept in bf16.
        {"name": "train 24x2048 bf16", "path": "train", "heads": 24, "n": 2048, "causal": False, "bf16": True, "reuse": False},
        # Scoring one 1024-token text with 12 heads.
        {"name": "forward 12x1024 causal", "path": "forward", "heads": 12, "n": 1024, "causal": True},
        # Long-sequence forward: 8 heads of 32768 tokens, no mask.
        {"name": "forward 8x32768", "path": "forward", "heads": 8, "n": 32768, "causal": False},
        # Interactive generation, host-launched, fp32 cache, early in a conversation: the smallest call.
        {"name": "step fp32 14/2 at 777", "path": "step", "n_head": 14, "n_kv": 2, "pos": 777, "quant": False, "paged": False},
        # Interactive generation as it is deployed: fp16 weights, int8 cache, 24 layers in one captured graph.
        {"name": "token int8 14/2 at 2000", "path": "token", "n_head": 14, "n_kv": 2, "pos": 2000, "quant": True, "layers": 24, "weights": "fp16"},
        # A serving step with a full batch over int8 paged caches.
        {"name": "batch 64 int8 14/2", "path": "batch", "n_head": 14, "n_kv": 2, "n_seq": 64, "ctx": 2048, "quant": True},
        # A serving step with a small batch over fp32 paged caches and a larger model's heads.
        {"name": "batch 16 fp32 32/4", "path": "batch", "n_head": 32, "n_kv": 4, "n_seq": 16, "ctx": 1500, "quant": False},
        # Question answering over very long documents, int8 cache.
        {"name": "long 8x131072 int8 32/4", "path": "long", "n_head": 32, "n_kv": 4, "n_seq": 8, "ctx": 131072, "quant": True},
        # The second turn of a conversation: 512 new tokens behind 1536 cached ones, int8 paged cache.
        {"name": "prefill 512+1536 int8", "path": "prefill", "n_head": 14, "n_kv": 2, "n_tok": 512, "pos0": 1536, "quant": True, "paged": True},
        # A long prompt's first chunk through a layer's attention half, fp32 cache, fp16 weights, ragged.
        {"name": "layer 1900+0 fp16", "path": "layer", "n_head": 14, "n_kv": 2, "n_tok": 1900, "pos0": 0, "quant": False, "paged": True,
         "weights": "fp16"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# query heads / KV heads of the decode and prefill cases: grouped as in the benchmark's configurations, and ungrouped
_HEADS = [(14, 2), (32, 4), (12, 12)]


def draw(rng):
    path = rng.choice(["train", "forward", "step", "token", "batch", "long", "prefill", "layer"])
    nh, nkv = rng.choice(_HEADS)
    quant, paged = rng.random() < 0.6, rng.random() < 0.5
    if path == "train":
        n = _log_int(rng, 128, 4096)
        bf16 = rng.random() < 0.4
        return {"path": path, "heads": _log_int(rng, 1, 48), "n": n, "causal": rng.random() < 0.7, "bf16": bf16,
                "reuse": not bf16 and rng.random() < 0.5}
    if path == "forward":
        n = _log_int(rng, 64, 32768)
        most = min(96, max(1, 8 * 32768 ** 2 // n ** 2))
        return {"path": path, "heads": _log_int(rng, 1, most), "n": n, "causal": rng.random() < 0.6}
    if path == "step":
        return {"path": path, "n_head": nh, "n_kv": nkv, "pos": _log_int(rng, 1, 4096) - 1, "quant": quant, "paged": paged}
    if path == "token":
        return {"path": path, "n_head": nh, "n_kv": nkv, "pos": _log_int(rng, 16, 4096) - 1, "quant": quant,
                "layers": rng.randint(4, 24), "weights": rng.choice(["fp16", "fp16", "fp32", "int8"])}
    if path == "batch":
        ctx = _log_int(rng, 64, 4096)
        return {"path": path, "n_head": nh, "n_kv": nkv, "n_seq": _log_int(rng, 2, 64 if nkv < 12 else 32), "ctx": ctx, "quant": quant}
    if path == "long":
        nh, nkv = rng.choice(_HEADS[:2])
        ctx = _log_int(rng, 8192, 131072)
        most = max(1, (604_000_000 if quant else 604_000_000 // 4) // (ctx * nkv * 144))
        return {"path": path, "n_head": nh, "n_kv": nkv, "n_seq": _log_int(rng, 1, min(8, most)), "ctx": ctx, "quant": quant}
    case = {"path": path, "n_head": nh, "n_kv": nkv, "n_tok": _log_int(rng, 16, 2048),
            "pos0": rng.choice([0, _log_int(rng, 1, 4096)]), "quant": quant, "paged": paged}
    if path == "layer":
        case["weights"] = rng.choice(["fp16", "fp32"])
    return case


def _normal(g, *shape):
    return torch.randn(*shape, device="cuda", generator=g)


def _table(g, n_log, first=0):
    return (torch.randperm(n_log, device="cuda", generator=g) + first).to(torch.int32)


def _cache(g, h, slots, n_kv, quant):
    """A cache of `slots` positions filled with N(0,1) rows, an int8 one by the library's own quantize-on-write."""
    c = la.KvCache(slots, n_kv, D, quant)
    kvd = n_kv * D
    for at in range(0, slots, 1 << 18):
        n = min(1 << 18, slots - at)
        if quant:
            rows = _normal(g, n, 2 * kvd)
            la.quantize_kv_batch(h, c, rows, at, n, 0, n_kv, D, 2 * kvd)
        else:
            c.k[at:at + n].normal_(generator=g)
            c.v[at:at + n].normal_(generator=g)
    return c


def _weights(g, kind, n_in, n_out):
    """(weights, column scales): activations of unit size stay of unit size through them."""
    if kind == "int8":
        codes = (_normal(g, n_in, n_out) * 32).round().clamp(-127, 127).to(torch.int32).reshape(n_in // 4, 4, n_out)
        packed = sum((codes[:, i] & 0xff) << (8 * i) for i in range(4)).to(torch.int32).contiguous()
        return packed, torch.full((n_out,), 1 / (32 * math.sqrt(n_in)), device="cuda")
    w = _normal(g, n_in, n_out) / math.sqrt(n_in)
    return (w.half() if kind == "fp16" else w), None


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    h = handle()
    h.set_option(_lib.OPT_BWD_REUSE_STAGED, int(case.get("reuse", False)))
    s = dict(case, h=h)
    path = case["path"]
    if path in ("train", "forward"):
        shape = (case["heads"], case["n"], D)
        h.reserve(fa.workspace_bytes(case["heads"], case["n"], path == "train"))
        s.update((x, _normal(g, *shape)) for x in ("q", "k", "v"))
        s["o"] = torch.empty(shape, device="cuda")
        if path == "train":
            s["do"] = _normal(g, *shape)
            s.update((x, torch.empty(shape, device="cuda")) for x in ("dq", "dk", "dv"))
            s.update((x, torch.empty(shape[:2], device="cuda")) for x in ("l", "delta"))
            if case["bf16"]:
                s.update((x, s[x].bfloat16()) for x in ("q", "k", "v"))
                s["dob"] = torch.empty_like(s["q"])
        return s
    nh, nkv, quant = case["n_head"], case["n_kv"], case["quant"]
    qd, kvd = nh * D, nkv * D
    row = qd + 2 * kvd
    s["stride"] = row
    if path == "step":
        slots = -(-(case["pos"] + 1) // BLOCK) * BLOCK
        s.update(c=_cache(g, h, slots, nkv, quant), qkv=_normal(g, row), out=torch.empty(qd, device="cuda"), pg=None, host=None)
        if case["paged"]:
            table = _table(g, slots // BLOCK)
            s.update(pg=la.Paging(table), host=table.cpu().numpy())
    elif path == "token":
        slots, n, kind = case["pos"] + 1, case["layers"], case["weights"]
        s["pos_dev"] = torch.full((1,), case["pos"], dtype=torch.int32, device="cuda")
        s["caches"] = [_cache(g, h, slots, nkv, quant) for _ in range(n)]
        s["w_qkv"] = [_weights(g, kind, qd, row) for _ in range(n)]
        s["w_out"] = [_weights(g, kind, qd, qd) for _ in range(n)]
        s["bias"] = _normal(g, n, row) * 0.1
        s["x"] = _normal(g, n, qd)
        s.update(qkv=torch.empty(n, row, device="cuda"), att=torch.empty(n, qd, device="cuda"), y=torch.empty(n, qd, device="cuda"))
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _token(s)  # first launches set kernel attributes: not inside a capture
        side.synchronize()
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"], stream=side):
            _token(s)
    elif path == "batch":
        n, ctx = case["n_seq"], case["ctx"]
        n_log = -(-ctx // BLOCK)
        # sequences of a running server: every length up to the largest, the longest among them
        pos = torch.randint(ctx // 4, ctx, (n,), device="cuda", generator=g, dtype=torch.int32)
        pos[0] = ctx - 1
        s.update(c=_cache(g, h, n * n_log * BLOCK, nkv, quant), pos=pos, pg=la.Paging(_table(g, n * n_log).reshape(n, n_log)),
                 qkv=_normal(g, n, row), out=torch.empty(n, qd, device="cuda"))
    elif path == "long":
        n, ctx = case["n_seq"], case["ctx"]
        s.update(c=_cache(g, h, n * ctx, nkv, quant), pos=torch.full((n,), ctx - 1, dtype=torch.int32, device="cuda"),
                 qkv=_normal(g, n, row), out=torch.empty(n, qd, device="cuda"))
    else:
        n_tok, pos0 = case["n_tok"], case["pos0"]
        slots = -(-(pos0 + n_tok) // BLOCK) * BLOCK
        h.reserve(la.prefill_workspace_bytes(n_tok, pos0 + n_tok, nh, nkv))
        s.update(c=_cache(g, h, slots, nkv, quant), pg=la.Paging(_table(g, slots // BLOCK)) if case["paged"] else None,
                 qkv=_normal(g, n_tok, row), out=torch.empty(n_tok, qd, device="cuda"))
        if path == "layer":
            s["x"], s["y"] = _normal(g, n_tok, qd), torch.empty(n_tok, qd, device="cuda")
            s["w_qkv"], s["w_out"] = _weights(g, case["weights"], qd, row)[0], _weights(g, case["weights"], qd, qd)[0]
            s["b_qkv"] = _normal(g, row) * 0.1
            for n in (row, qd):
                h.reserve(int(_lib.lib().mx230_gemm_workspace_bytes(n_tok, n, qd, int(case["weights"] == "fp16"))))
    return s


def _cache_state(c):
    return [c.k, c.v] + ([c.ks, c.vs, c.kb, c.vb] if c.quant else [])


def _token(s):
    h, nh, nkv = s["h"], s["n_head"], s["n_kv"]
    for i, c in enumerate(s["caches"]):
        (wq, sq), (wo, so) = s["w_qkv"][i], s["w_out"][i]
        la.qkv_rope_kvwrite(h, s["qkv"][i], s["x"][i], wq, s["bias"][i], s["pos_dev"], c, nh, nkv, THETA, w_scales=sq)
        la.attn_decode_dyn(h, s["att"][i], s["qkv"][i], c, s["pos_dev"], nh, nkv, D)
        if so is None:
            la.gemv(h, s["y"][i], s["att"][i], wo)
        else:
            la.gemv_int8(h, s["y"][i], s["att"][i], wo, so)


def run(s):
    h, path = s["h"], s["path"]
    if path == "train":
        n, causal = s["n"], s["causal"]
        if s["bf16"]:
            fa.run_flash_bf16(h, s["q"], s["k"], s["v"], s["o"], s["l"], n, causal)
            fa.run_preprocess(h, s["do"], s["o"], s["delta"], n)
            fa.cast_bf16(h, s["do"], s["dob"])
            fa.run_bwd_flash_bf16(h, s["q"], s["k"], s["v"], s["dob"], s["l"], s["delta"], s["dq"], s["dk"], s["dv"], n, causal)
        else:
            fa.run_flash_lse(h, s["q"], s["k"], s["v"], s["o"], s["l"], n, causal)
            fa.run_preprocess(h, s["do"], s["o"], s["delta"], n)
            fa.run_bwd_flash(h, s["q"], s["k"], s["v"], s["do"], s["l"], s["delta"], s["dq"], s["dk"], s["dv"], n, causal)
        return [s[x] for x in ("o", "l", "delta", "dq", "dk", "dv")]
    if path == "forward":
        fa.run_flash(h, s["q"], s["k"], s["v"], s["o"], s["n"], s["causal"])
        return s["o"]
    nh, nkv = s["n_head"], s["n_kv"]
    if path == "token":
        s["graph"].replay()
        return [s["y"], s["att"], s["qkv"]] + [c.k for c in s["caches"]]
    if path == "long":
        la.attn_decode_slab(h, s["out"], s["qkv"], s["c"], s["pos"], s["n_seq"], nh, nkv, D, s["ctx"], s["stride"], nh * D)
        return s["out"]
    if path == "step":
        la.decode_step(h, s["out"], s["qkv"], s["c"], s["pos"], nh, nkv, D, THETA, s["pg"], s["host"])
        return [s["out"], s["qkv"]] + _cache_state(s["c"])
    if path == "batch":
        la.batched_step(h, s["out"], s["qkv"], s["c"], s["pos"], s["n_seq"], nh, nkv, D, THETA, s["pg"], s["stride"], nh * D)
        return [s["out"], s["qkv"]] + _cache_state(s["c"])
    if path == "prefill":
        la.prefill_step(h, s["out"], s["qkv"], s["c"], s["pos0"], s["n_tok"], nh, nkv, D, THETA, s["stride"], nh * D, s["pg"])
        return [s["out"], s["qkv"]] + _cache_state(s["c"])
    la.prefill_layer_attention(h, s["y"], s["x"], s["w_qkv"], s["b_qkv"], s["w_out"], None, s["qkv"], s["out"], s["c"], s["pos0"],
                               s["n_tok"], nh, nkv, D, THETA, s["pg"])
    return [s["y"], s["out"], s["qkv"]] + _cache_state(s["c"])


def work(case):
    path = case["path"]
    if path in ("train", "forward"):
        e = case["heads"] * case["n"]                       # rows
        fwd = 4.0 * e * case["n"] * D / (2 if case["causal"] else 1)
        if path == "forward":
            return {"bytes": 4 * 4 * e * D, "flops": fwd}
        ins = 3 * 2 + 4 if case["bf16"] else 4 * 4          # q, k, v and dO
        return {"bytes": e * D * (ins + 4 * 4) + 2 * 4 * e, "flops": 3.5 * fwd}
    nh, nkv, quant = case["n_head"], case["n_kv"], case["quant"]
    qd, kvd = nh * D, nkv * D
    row = qd + 2 * kvd
    key = nkv * (2 * (D + 8) if quant else 2 * D * 4)       # bytes of one cached position
    per_tok = 4 * (row + qd + qd + kvd) + key               # qkv in, rotated q and k out, attention row out, cache row out
    attend = 4.0 * qd                                       # operations of one query row on one key
    if path == "step":
        return {"bytes": case["pos"] * key + per_tok, "flops": attend * (case["pos"] + 1)}
    if path == "token":
        n, size = case["layers"], {"fp32": 4, "fp16": 2, "int8": 1}[case["weights"]]
        w = qd * (row + qd)
        return {"bytes": n * (w * size + case["pos"] * key + per_tok + 8 * qd), "flops": n * (2.0 * w + attend * (case["pos"] + 1))}
    if path == "batch":
        keys = case["n_seq"] * case["ctx"] * 0.625          # positions are spread evenly over [ctx / 4, ctx)
        return {"bytes": keys * key + case["n_seq"] * per_tok, "flops": attend * keys}
    if path == "long":
        keys = case["n_seq"] * case["ctx"]
        return {"bytes": keys * key + case["n_seq"] * 8 * qd, "flops": attend * keys}
    n_tok, pos0 = case["n_tok"], case["pos0"]
    pairs = n_tok * pos0 + n_tok * (n_tok + 1) / 2
    b, f = pos0 * key + n_tok * per_tok, attend * pairs
    if path == "layer":
        w = qd * (row + qd)
        b += w * (2 if case["weights"] == "fp16" else 4) + n_tok * 8 * qd
        f += 2.0 * n_tok * w
    return {"bytes": b, "flops": f}


def tolerance(case):
    """Measured against the same sums in 64 bits. bf16 operands on the tensor cores: 2e-3 to 4.6e-3 in the 2-norm (gradients the
    most), single values up to 0.15 of the root mean square. fp32 caches: 2e-7. int8 caches: 3e-6 to 5e-6, and a rotated q that
    rounds the other way moves one of its int8 codes, and with it a head's row by up to 3e-3."""
    path, quant = case["path"], case.get("quant", False)
    if path in ("train", "forward", "prefill", "layer"):
        return {"rel": 1e-2, "max": 0.4, "differ": 1e-3}
    return {"rel": 1e-4, "max": 1e-2, "differ": 1e-4} if quant else {"rel": 1e-5, "max": 1e-3}

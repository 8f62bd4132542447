"""The fused prefill step (RoPE, KV write and staging in one launch) against the separate entry points it stands for, and
the forms of the forward kernel that a prefill call can take, at the edges of their tiles."""
import numpy as np
import pytest
import torch

import oracle
from mx230_b200 import _lib
from mx230_b200 import llm_attention as la

pytestmark = pytest.mark.gpu
THETA = 1e6


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def filled_cache(handle, slots, nkv, quant, affine, seed):
    c = la.KvCache(slots, nkv, 64, quant, affine)
    rows = dev(oracle.normal((slots, 2 * nkv * 64), seed, 0))
    if quant:
        la.quantize_kv_batch(handle, c, rows, 0, slots, 0, nkv, 64, 2 * nkv * 64)
    else:
        c.k.copy_(rows[:, :nkv * 64])
        c.v.copy_(rows[:, nkv * 64:])
    return c


def arrays(c):
    return [x for x in (c.k, c.v, c.ks, c.vs, c.kb, c.vb) if x is not None] if c.quant else [c.k, c.v]


@pytest.mark.parametrize("quant,affine,exact", [(False, True, False), (True, True, False), (True, False, False), (True, True, True)])
@pytest.mark.parametrize("nh,nkv,n_tok,pos0,paged,rope", [
    (14, 2, 1, 0, False, True), (14, 2, 5, 130, True, True), (12, 12, 129, 127, True, True), (18, 2, 70, 333, False, True),
    (4, 1, 640, 3, True, False), (32, 4, 257, 1000, True, True),
])
def test_step_equals_separate_calls(handle, quant, affine, exact, nh, nkv, n_tok, pos0, paged, rope):
    qd, stride = nh * 64, (nh + 2 * nkv) * 64 + 8
    slots = -(-(pos0 + n_tok) // 16) * 16
    pg = la.Paging(dev(np.random.default_rng(1).permutation(slots // 16).astype(np.int32))) if paged else None
    qkv = dev(oracle.normal((n_tok, stride), 701, 0))
    qkv_f = qkv.clone()
    c, c_f = (filled_cache(handle, slots, nkv, quant, affine, 702) for _ in range(2))
    out, out_f = (torch.full((n_tok, qd + 4), 7.0, device="cuda") for _ in range(2))
    handle.reserve(la.prefill_workspace_bytes(n_tok, pos0 + n_tok, nh, nkv))
    handle.set_option(_lib.OPT_Q8_SCORE_MODE, _lib.Q8_SCORE_EXACT if exact else _lib.Q8_SCORE_REF)
    try:
        if rope:
            la.rope_batch(handle, qkv, pos0, n_tok, nh, nkv, 64, stride, THETA)
        if quant:
            la.quantize_kv_batch(handle, c, qkv, pos0, n_tok, qd, nkv, 64, stride, pg)
        else:
            la.copy_kv_batch(handle, c, qkv, pos0, n_tok, qd, nkv * 64, stride, pg)
        la.attn_prefill(handle, out, qkv, c, pos0, n_tok, nh, nkv, stride, qd + 4, pg)
        la.prefill_step(handle, out_f, qkv_f, c_f, pos0, n_tok, nh, nkv, 64, THETA, stride, qd + 4, pg, use_rope=rope)
        handle.check_status()
    finally:
        handle.set_option(_lib.OPT_Q8_SCORE_MODE, _lib.Q8_SCORE_REF)
    assert torch.equal(qkv, qkv_f)
    for a, b in zip(arrays(c), arrays(c_f)):
        assert torch.equal(a, b)
    assert torch.equal(out, out_f)


def scores64(qkv, c, nh, nkv, n_keys, quant):
    """Scores in 64 bits; over an int8 cache from the codes, as the score mode defines them."""
    q = qkv[:, :nh * 64].reshape(-1, nh, 64).double()
    k = c.k[:n_keys].reshape(n_keys, nkv, 64).double()
    v = c.v[:n_keys].reshape(n_keys, nkv, 64).double()
    if quant:
        q32 = qkv[:, :nh * 64].reshape(-1, nh, 64)
        amax = q32.abs().amax(-1, keepdim=True)
        q = torch.round(q32 * (127.0 / amax)).clamp(-127, 127).double() * (amax / 127.0).double()
        k = k * c.ks[:n_keys, :, None].double() + c.kb[:n_keys, :, None].double()
        v = v * c.vs[:n_keys, :, None].double() + c.vb[:n_keys, :, None].double()
    rep = nh // nkv
    return torch.einsum("thd,khd->htk", q, k.repeat_interleave(rep, 1)) * 0.125, v.repeat_interleave(rep, 1)


@pytest.mark.parametrize("quant", [False, True])
@pytest.mark.parametrize("scale", [1.0, 40.0])   # 40: scores beyond the bound of the max-free loop
@pytest.mark.parametrize("nh,nkv,n_tok,pos0", [
    (2, 1, 1, 0), (2, 1, 128, 0), (3, 3, 129, 1), (2, 2, 100, 200), (14, 2, 257, 130), (3, 1, 640, 129),   # few items: 64-row form
    (14, 2, 700, 300), (14, 2, 1200, 0), (14, 2, 1410, 77),          # key-split form, the last one with several items per CTA
    (40, 8, 1024, 0),                                                # pair form
])
def test_forms_and_edges(handle, quant, scale, nh, nkv, n_tok, pos0):
    """Every form against 64-bit softmax.  The probabilities and V are rounded to bf16 (2^-9 each, relative): a row is an
    average of values of size about 1 with an error below 2 * 2^-9 * max|v|, max|v| < 5.5 here.  fp32 caches: q and k are
    rounded as well, which moves a score by about 2^-9 |q||k| / 8 (sd 2^-9 * scale), and with it a probability by that
    factor: 1e-2 at scale 1.  At scale 40 the softmax is close to one-hot and such a score error can swap the leading keys,
    so only int8 scores (exact in bf16) are compared value by value there; for fp32 the row must be a convex combination."""
    n_keys = pos0 + n_tok
    stride = (nh + 2 * nkv) * 64
    c = filled_cache(handle, n_keys, nkv, quant, True, 712)
    qkv = dev(oracle.normal((n_tok, stride), 711, 0)) * scale
    out = torch.empty(n_tok, nh * 64, device="cuda")
    handle.reserve(la.prefill_workspace_bytes(n_tok, n_keys, nh, nkv))
    la.attn_prefill(handle, out, qkv, c, pos0, n_tok, nh, nkv, stride, nh * 64)
    handle.check_status()
    s, v = scores64(qkv, c, nh, nkv, n_keys, quant)
    mask = torch.arange(n_keys, device="cuda")[None, :] > torch.arange(n_tok, device="cuda")[:, None] + pos0
    p = torch.softmax(s.masked_fill(mask, -float("inf")), -1)
    want = torch.einsum("htk,khd->thd", p, v).reshape(n_tok, nh * 64)
    got = out.double()
    assert torch.isfinite(got).all()
    if quant or scale == 1.0:
        assert (got - want).abs().max() <= 4e-2
        assert (got - want).abs().mean() / want.abs().mean() <= 6e-3
    else:
        lo, hi = v.amin(), v.amax()
        assert got.min() >= lo * (1 + 2.0 ** -7) and got.max() <= hi * (1 + 2.0 ** -7)


@pytest.mark.parametrize("nh,nkv,n_tok,pos0", [(14, 2, 1900, 0), (14, 2, 1450, 500), (32, 4, 1024, 0)])   # key-split, over 148 items
@pytest.mark.parametrize("every,first", [(3, 1), (2, 0), (5, 2)])
def test_heads_inside_and_outside_the_bound_in_one_call(handle, nh, nkv, n_tok, pos0, every, first):
    """int8 scores, several items per SM, some heads beyond the bound of the max-free loop: an SM goes from an item of one loop
    to an item of the other.  Against 64-bit softmax (bounds of the test above), and a head inside the bound has the same
    bits in a call of its own; every pass gives the same bits."""
    n_keys, stride = pos0 + n_tok, (nh + 2 * nkv) * 64
    c = filled_cache(handle, n_keys, nkv, True, True, 722)
    qkv = dev(oracle.normal((n_tok, stride), 721, 0))
    beyond = [h for h in range(nh) if h % every == first]
    for h in beyond:
        qkv[:, h * 64:(h + 1) * 64] *= 40
    out, again = torch.empty(n_tok, nh * 64, device="cuda"), torch.empty(n_tok, nh * 64, device="cuda")
    handle.reserve(la.prefill_workspace_bytes(n_tok, n_keys, nh, nkv))
    la.attn_prefill(handle, out, qkv, c, pos0, n_tok, nh, nkv, stride, nh * 64)
    for _ in range(10):
        la.attn_prefill(handle, again, qkv, c, pos0, n_tok, nh, nkv, stride, nh * 64)
        assert torch.equal(out, again)
    handle.check_status()
    mask = torch.arange(n_keys, device="cuda")[None, :] > torch.arange(n_tok, device="cuda")[:, None] + pos0
    for g in range(nkv):
        rep = nh // nkv
        q = qkv[:, g * rep * 64:(g + 1) * rep * 64]
        c1 = la.KvCache(n_keys, 1, 64, True)
        for x in ("k", "v"):
            getattr(c1, x).copy_(getattr(c, x)[:, g * 64:(g + 1) * 64])
        for x in ("ks", "vs", "kb", "vb"):
            getattr(c1, x).copy_(getattr(c, x)[:, g:g + 1])
        s, v = scores64(q, c1, rep, 1, n_keys, True)
        want = torch.einsum("htk,khd->thd", torch.softmax(s.masked_fill(mask, -float("inf")), -1), v).reshape(n_tok, rep * 64)
        got = out[:, g * rep * 64:(g + 1) * rep * 64]
        assert (got.double() - want).abs().max() <= 4e-2
        assert (got.double() - want).abs().mean() / want.abs().mean() <= 6e-3
        for h in range(rep):
            if g * rep + h not in beyond:
                one = torch.empty(n_tok, 64, device="cuda")
                la.attn_prefill(handle, one, q[:, h * 64:(h + 1) * 64].contiguous(), c1, pos0, n_tok, 1, 1, 64, 64)
                assert torch.equal(one, got[:, h * 64:(h + 1) * 64]), f"head {g * rep + h}"
    handle.check_status()


@pytest.mark.parametrize("quant", [False, True])
@pytest.mark.parametrize("nh", [12284, 12286, 12288])   # with two K/V heads: the most whose norms a CTA keeps is 12286
def test_very_many_heads(handle, quant, nh):
    nkv, n_tok, pos0 = 2, 3, 5
    n_keys, stride = pos0 + n_tok, (nh + 2 * nkv) * 64
    c = filled_cache(handle, n_keys, nkv, quant, True, 732)
    qkv = dev(oracle.normal((n_tok, stride), 731, 0))
    out = torch.empty(n_tok, nh * 64, device="cuda")
    handle.reserve(la.prefill_workspace_bytes(n_tok, n_keys, nh, nkv))
    la.attn_prefill(handle, out, qkv, c, pos0, n_tok, nh, nkv, stride, nh * 64)
    handle.check_status()
    s, v = scores64(qkv, c, nh, nkv, n_keys, quant)
    mask = torch.arange(n_keys, device="cuda")[None, :] > torch.arange(n_tok, device="cuda")[:, None] + pos0
    want = torch.einsum("htk,khd->thd", torch.softmax(s.masked_fill(mask, -float("inf")), -1), v).reshape(n_tok, nh * 64)
    assert (out.double() - want).abs().max() <= 4e-2 and (out.double() - want).abs().mean() / want.abs().mean() <= 6e-3   # as above

"""The prefill step followed by the output projection in one call: attention leaves its rows in fp16 for the projection, which
gives the bits of the two calls in turn (the same rounding, the same products)."""
import functools

import numpy as np
import pytest
import torch

import oracle
from mx230_b200 import llm_attention as la
from mx230_b200._lib import (ERR_INVALID_ARG, ERR_UNSUPPORTED, OPT_Q8_SCORE_MODE, Q8_SCORE_EXACT, Q8_SCORE_REF, Mx230Error, check,
                             lib, ptr)

pytestmark = pytest.mark.gpu
THETA = 1e6


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@functools.lru_cache(maxsize=None)
def normal(shape, seed):
    return oracle.normal(shape, seed, 0)


def caches(c):
    return [x for x in (c.k, c.v, c.ks, c.vs, c.kb, c.vb) if x is not None] if c.quant else [c.k, c.v]


# query tiles of 128 rows: one row, either side of a tile, an odd number of tiles; both forms of the forward (40 heads: pair
# form); output columns by whole (stored by TMA) and ragged 64-column chunks; 1900 rows: 15 row tiles of the projection, the last
# ragged.  Caches in order and paged; int8 in both score modes.
@pytest.mark.parametrize("cache", ["fp32", "int8", "int8 exact"])
@pytest.mark.parametrize("paged", [False, True])
@pytest.mark.parametrize("nh,nkv,n_tok,pos0,n_out", [
    (14, 2, 1, 0, 896), (14, 2, 127, 5, 72), (12, 12, 128, 0, 768), (14, 2, 129, 300, 896), (14, 2, 1900, 44, 896),
    (40, 8, 2050, 0, 200),
])
def test_step_with_projection_equals_the_calls_in_turn(handle, cache, paged, nh, nkv, n_tok, pos0, n_out):
    quant = cache != "fp32"
    handle.set_option(OPT_Q8_SCORE_MODE, Q8_SCORE_EXACT if cache == "int8 exact" else Q8_SCORE_REF)
    try:
        _equals_the_calls_in_turn(handle, quant, paged, nh, nkv, n_tok, pos0, n_out)
    finally:
        handle.set_option(OPT_Q8_SCORE_MODE, Q8_SCORE_REF)


def _equals_the_calls_in_turn(handle, quant, paged, nh, nkv, n_tok, pos0, n_out):
    qd, row, e = nh * 64, (nh + 2 * nkv) * 64, 128
    x = dev(normal((n_tok, e), 811))
    w_qkv = dev((normal((e, row), 812) / np.sqrt(e)).astype(np.float16))
    w_proj = dev((normal((qd, n_out), 813) / np.sqrt(qd)).astype(np.float16))
    b_proj = dev(normal((n_out,), 814))
    old = dev(normal((max(pos0, 1), 2 * nkv * 64), 815))
    handle.reserve(la.prefill_workspace_bytes(n_tok, pos0 + n_tok, nh, nkv))
    blocks = -(-(pos0 + n_tok) // la.KV_BLOCK)
    table = np.random.default_rng(5).permutation(blocks).astype(np.int32)
    pg = la.Paging(dev(table)) if paged else None
    at = np.arange(pos0)   # the cache rows of the old positions
    at = dev(table[at // la.KV_BLOCK] * la.KV_BLOCK + at % la.KV_BLOCK).long() if paged else slice(0, pos0)
    got = []
    for fused in (False, True):
        c = la.KvCache(blocks * la.KV_BLOCK, nkv, 64, quant)
        if quant:
            la.quantize_kv_batch(handle, c, old, 0, pos0, 0, nkv, 64, 2 * nkv * 64, pg)
        else:
            c.k[at], c.v[at] = old[:pos0, :nkv * 64], old[:pos0, nkv * 64:]
        qkv, attn = torch.zeros(n_tok, row, device="cuda"), torch.full((n_tok, qd), float("nan"), device="cuda")
        y = torch.full((n_tok, n_out), float("nan"), device="cuda")
        if fused:
            la.prefill_layer_attention(handle, y, x, w_qkv, None, w_proj, b_proj, qkv, attn, c, pos0, n_tok, nh, nkv, 64, THETA, pg)
        else:
            la.gemm(handle, qkv, x, w_qkv)
            la.prefill_step(handle, attn, qkv, c, pos0, n_tok, nh, nkv, 64, THETA, row, qd, pg)
            la.gemm(handle, y, attn, w_proj, b_proj)
        handle.check_status()
        got.append([y, attn, qkv] + caches(c))
    assert not torch.isnan(got[1][0]).any()
    for a, b in zip(*got):
        assert torch.equal(a, b)


def test_step_with_projection_rejects_bad_arguments(handle):
    c = la.KvCache(16, 2, 64, False)
    qkv, out = torch.zeros(4, 18 * 64, device="cuda"), torch.zeros(4, 14 * 64, device="cuda")
    w, y = torch.zeros(14 * 64, 64, dtype=torch.float16, device="cuda"), torch.full((4, 64), 7.0, device="cuda")
    cache = (ptr(c.k), ptr(c.v), None, None, None, None, None, None)

    def call(y_=ptr(y), n_out=64, head_dim=64):
        check(lib().mx230_prefill_step_proj(handle._h, None, y_, ptr(w), None, n_out, ptr(out), ptr(qkv), *cache, 0, 4, 14, 2,
                                            head_dim, 1, THETA, 18 * 64, 14 * 64, None, 0))
    for kw, code in [(dict(y_=None), ERR_INVALID_ARG), (dict(n_out=12), ERR_UNSUPPORTED), (dict(n_out=0), ERR_UNSUPPORTED),
                     (dict(head_dim=32), ERR_UNSUPPORTED), (dict(y_=y.data_ptr() + 4), ERR_INVALID_ARG)]:
        with pytest.raises(Mx230Error) as err:
            call(**kw)
        assert err.value.code == code
    assert (y == 7.0).all() and (qkv == 0).all()

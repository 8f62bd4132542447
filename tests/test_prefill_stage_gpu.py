"""The two grids of the prefill staging kernel (128 CTAs, 256 where tokens or cached keys would take more than one round): the
fused step against the separate entry points either side of both lines.  The step stages cached keys and new tokens apart,
plain attention takes all keys from the cache, so the two are staged by different grids and warps here."""
import numpy as np
import pytest
import torch

import oracle
from mx230_b200 import llm_attention as la
from tests.test_prefill_step_gpu import THETA, arrays, dev, filled_cache

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quant", [False, True])
@pytest.mark.parametrize("nh,nkv,n_tok,pos0", [
    (2, 2, 512, 0), (2, 2, 513, 5),                 # tokens: one round of 128 CTAs, one more
    (14, 2, 3, 4096), (14, 2, 3, 4097),             # cached keys: 65536 threads, eight more
    (12, 12, 20, 682), (12, 12, 20, 683), (3, 1, 1, 31), (21, 3, 2100, 1333),   # 21 + 2 * 3 heads: two rounds of five a warp
])
def test_step_equals_separate_calls(handle, quant, nh, nkv, n_tok, pos0):
    qd, stride = nh * 64, (nh + 2 * nkv) * 64
    slots = -(-(pos0 + n_tok) // 16) * 16
    pg = la.Paging(dev(np.random.default_rng(2).permutation(slots // 16).astype(np.int32)))
    qkv = dev(oracle.normal((n_tok, stride), 711, 0))
    qkv_f = qkv.clone()
    c, c_f = (filled_cache(handle, slots, nkv, quant, True, 712) for _ in range(2))
    out, out_f = (torch.full((n_tok, qd), float("nan"), device="cuda") for _ in range(2))
    handle.reserve(la.prefill_workspace_bytes(n_tok, pos0 + n_tok, nh, nkv))
    la.rope_batch(handle, qkv, pos0, n_tok, nh, nkv, 64, stride, THETA)
    if quant:
        la.quantize_kv_batch(handle, c, qkv, pos0, n_tok, qd, nkv, 64, stride, pg)
    else:
        la.copy_kv_batch(handle, c, qkv, pos0, n_tok, qd, nkv * 64, stride, pg)
    la.attn_prefill(handle, out, qkv, c, pos0, n_tok, nh, nkv, stride, qd, pg)
    la.prefill_step(handle, out_f, qkv_f, c_f, pos0, n_tok, nh, nkv, 64, THETA, stride, qd, pg)
    handle.check_status()
    assert torch.equal(qkv, qkv_f) and torch.equal(out, out_f) and not torch.isnan(out).any()
    for a, b in zip(arrays(c), arrays(c_f)):
        assert torch.equal(a, b)

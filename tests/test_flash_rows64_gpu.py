"""Forward with 64-row items (calls whose 64-row items fit the SMs at once) against the other forms, which calls with more heads
take: a head inside the bound has the same bits in either, a head beyond it (its own max per softmax group) the same rows up to
the rounding of P.  Sizes are the edges of 64-row tiles, of 128-key tiles and of rounds of four key tiles."""
import pytest
import torch

from mx230_b200 import flash_attention as fa
from mx230_b200 import llm_attention as la

pytestmark = pytest.mark.gpu


def many(n):
    """Heads that are too many for 64-row items."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return sms // (-(-n // 64)) + 1


# P is rounded to bf16 (2^-9 relative) against another reference in either form: rows differ by less than 2 * 2^-9 * max|v| (< 5.5)
ROWS = 2.2e-2


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 128, 129, 255, 300, 511, 513, 700, 1024, 1921, 2050, 2177])
def test_equals_the_other_forms(handle, n, causal, bf16):
    heads = many(n)
    g = torch.Generator(device="cuda")
    g.manual_seed(31)
    q, k, v = (torch.randn(heads, n, 64, device="cuda", generator=g) for _ in range(3))
    q[1] *= 40
    if bf16:
        q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    run = fa.run_flash_bf16 if bf16 else fa.run_flash_lse
    handle.reserve(fa.workspace_bytes(heads, n, False))
    o, l = torch.full((heads, n, 64), float("nan"), device="cuda"), torch.full((heads, n), float("nan"), device="cuda")
    run(handle, q, k, v, o, l, n, causal)
    few = 2 if n <= 2048 else 1
    o2, l2 = torch.full((few, n, 64), float("nan"), device="cuda"), torch.full((few, n), float("nan"), device="cuda")
    run(handle, q[:few], k[:few], v[:few], o2, l2, n, causal)
    handle.check_status()
    assert torch.isfinite(o2).all() and torch.isfinite(l2).all()
    if not bf16 or n > 1920:       # (shorter bf16 calls have no bound and take the general loop)
        assert torch.equal(o[0], o2[0]) and torch.equal(l[0], l2[0])
    assert (o[:few] - o2).abs().max() <= ROWS and (l[:few] - l2).abs().max() <= 1e-3


@pytest.mark.parametrize("quant", [False, True])
@pytest.mark.parametrize("n_tok,pos0", [(1, 0), (1, 127), (1, 128), (64, 64), (65, 0), (65, 511), (130, 700), (300, 1500), (16, 4000),
                                         (64, 1217), (65, 1300), (1, 1535), (1, 1536), (257, 1280)])
def test_prefill_equals_the_other_forms(handle, quant, n_tok, pos0):
    """With the causal offset, over both score sources; heads 1 and up share K/V head 0 and are copies of head 0 (head 2 scaled beyond
    the bound), so that one call of the general size holds the heads of the small one."""
    nh, n_keys = many(n_tok), pos0 + n_tok
    g = torch.Generator(device="cuda")
    g.manual_seed(32)
    c = la.KvCache(n_keys, 1, 64, quant)
    kv = torch.randn(n_keys, 128, device="cuda", generator=g)
    if quant:
        la.quantize_kv_batch(handle, c, kv, 0, n_keys, 0, 1, 64, 128)
    else:
        c.k.copy_(kv[:, :64]), c.v.copy_(kv[:, 64:])
    q = torch.randn(n_tok, 1, 64, device="cuda", generator=g).repeat(1, nh, 1)
    q[:, 2 % nh] *= 40
    handle.reserve(la.prefill_workspace_bytes(n_tok, n_keys, nh, 1))
    out = torch.full((n_tok, nh * 64), float("nan"), device="cuda")
    la.attn_prefill(handle, out, q.reshape(n_tok, nh * 64).contiguous(), c, pos0, n_tok, nh, 1, nh * 64, nh * 64)
    for h, same in ((0, True), (2 % nh, False)):
        one = torch.full((n_tok, 64), float("nan"), device="cuda")
        la.attn_prefill(handle, one, q[:, h].contiguous(), c, pos0, n_tok, 1, 1, 64, 64)
        handle.check_status()
        assert torch.isfinite(one).all()
        want = out[:, h * 64:(h + 1) * 64]
        assert torch.equal(one, want) if same else (one - want).abs().max() <= ROWS

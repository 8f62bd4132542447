"""Fused backward, several items per SM: the owned K and V tiles of the next item arrive while the current one still runs, K in
the place of a streamed tile.  Items of one, two and three streamed tiles in every order a CTA can meet them, and longer ones."""
import pytest
import torch

from mx230_b200 import _lib
from mx230_b200 import flash_attention as fa

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("heads,n,causal", [
    (500, 128, False), (500, 100, True),   # one-tile items only, three to four per SM
    (400, 200, True), (300, 256, False),   # two and one
    (200, 384, True), (160, 300, False),   # three, two, one; ragged
    (60, 1100, True),                      # nine to one
])
def test_every_head_equals_itself_alone(handle, heads, n, causal, bf16):
    """dK and dV of a head are sums in the order of its query tiles, whichever CTA has them: the bits of the head in a call of
    its own (where no SM has a second item).  dQ's partial sums (one per key tile, at most 9) arrive in any order: two such sums
    differ by at most 2 * 9 * 2^-24 of the sum of the terms' sizes, which 16 times the largest |dQ| bounds here."""
    g = torch.Generator(device="cuda")
    g.manual_seed(31)
    q, k, v, do = (torch.randn(heads, n, 64, device="cuda", generator=g) for _ in range(4))
    fwd = fa.run_flash_bf16 if bf16 else fa.run_flash_lse
    bwd = fa.run_bwd_flash_bf16 if bf16 else fa.run_bwd_flash
    if bf16:
        q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    d_in = do.bfloat16() if bf16 else do
    handle.reserve(fa.workspace_bytes(heads, n, True))

    o, (l, delta) = torch.empty_like(do), (torch.empty(heads, n, device="cuda") for _ in range(2))
    fwd(handle, q, k, v, o, l, n, causal)
    fa.run_preprocess(handle, do, o, delta, n)

    def grads(s):   # of these heads, from the same L and Delta
        out = [torch.full_like(do[s], float("nan")) for _ in range(3)]
        bwd(handle, q[s], k[s], v[s], d_in[s], l[s], delta[s], *out, n, causal)
        handle.check_status()
        return out

    dq, dk, dv = grads(slice(0, heads))
    for h in sorted({0, 1, heads // 3, 147, 148, heads - 2, heads - 1} & set(range(heads))):
        aq, ak, av = grads(slice(h, h + 1))
        assert torch.equal(dk[h], ak[0]) and torch.equal(dv[h], av[0]), f"head {h}"
        assert (dq[h] - aq[0]).abs().max() <= 2 * 9 * 2 ** -24 * 16 * aq.abs().max(), f"head {h}"
    for h in (0, heads - 1):   # against 64-bit gradients: operands rounded to bf16, as in the backward's other tests
        x = [t[h].double().requires_grad_() for t in (q, k, v)]
        s = x[0] @ x[1].T * 0.125
        if causal:
            s = s.masked_fill(torch.triu(torch.ones(n, n, dtype=torch.bool, device="cuda"), 1), -float("inf"))
        want = torch.autograd.grad(torch.softmax(s, -1) @ x[2], x, do[h].double())
        for got, w in zip((dq[h], dk[h], dv[h]), want):
            assert (got.double() - w).norm() / w.norm() <= 1e-2


def test_profile_has_every_launch(handle):
    """The kernel that clears dQ where no staging launch does is in the profile; the launch count leaves it out, as it would the
    memset in whose place it stands."""
    heads, n = 3, 200
    x = [torch.randn(heads, n, 64, device="cuda") for _ in range(4)]
    b = [t.bfloat16() for t in x]
    o, dq, dk, dv = (torch.empty_like(x[0]) for _ in range(4))
    l, delta = (torch.empty(heads, n, device="cuda") for _ in range(2))

    def counted(f):
        l0 = handle.launches
        handle.profile_reset()
        handle.profile_enable(True)
        f()
        handle.profile_enable(False)
        prof = {k: v[0] for k, v in handle.profile_read().items()}
        assert handle.launches - l0 == sum(prof.values()) - prof.get("zero_kernel", 0)
        return prof

    fa.run_flash_bf16(handle, *b[:3], o, l, n, True)
    fa.run_preprocess(handle, x[3], o, delta, n)
    got = counted(lambda: fa.run_bwd_flash_bf16(handle, *b, l, delta, dq, dk, dv, n, True))
    assert got == {"zero_kernel": 1, "bwd_fused_kernel": 1}
    handle.reserve(fa.workspace_bytes(heads, n, True))
    handle.set_option(_lib.OPT_BWD_REUSE_STAGED, 1)
    try:
        fa.run_flash_lse(handle, *x[:3], o, l, n, True)
        fa.run_preprocess(handle, x[3], o, delta, n)
        got = counted(lambda: fa.run_bwd_flash(handle, *x, l, delta, dq, dk, dv, n, True))
    finally:
        handle.set_option(_lib.OPT_BWD_REUSE_STAGED, 0)
    assert got == {"zero_kernel": 1, "bwd_fused_kernel": 1}
    got = counted(lambda: fa.run_bwd_flash(handle, *x, l, delta, dq, dk, dv, n, True))
    assert got == {"cast_bf16_kernel": 1, "bwd_fused_kernel": 1}
    handle.check_status()

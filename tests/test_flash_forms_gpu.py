"""Forward over operands the caller staged (bf16): the form of the kernel, its max-free loop (from 16 key tiles per row on,
where a pass over Q and K bounds a head's scores) and its general loop, mixed among the heads of one call."""
import pytest
import torch

from mx230_b200 import flash_attention as fa

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("heads,n", [(3, 1920), (3, 1921), (3, 2177), (1, 4096),     # 64-row form
                                     (17, 1024), (8, 1921), (10, 1920), (9, 2177),   # key-split (the last two: causal, over 148 items)
                                     (40, 2050)])                                    # pair form
def test_bf16_forward_modes(handle, heads, n, causal):
    """bf16 operands are exact, so scores differ from 64 bits by fp32 rounding only (2^-24 * 64 * |q||k|/8 < 2e-3 at the
    largest scale here, below 1e-5 at scale 1): what remains is P in bf16, 2^-9 relative per probability, which moves a row by
    less than 2 * 2^-9 * max|v| (max|v| < 5.5), and ln of an fp32 sum."""
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    q, k, v = (torch.randn(heads, n, 64, device="cuda", generator=g) for _ in range(3))
    q[1::3] *= 30          # scores beyond the bound: these heads take the general loop
    q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    o, l = torch.empty(heads, n, 64, device="cuda"), torch.full((heads, n), float("nan"), device="cuda")
    fa.run_flash_bf16(handle, q, k, v, o, l, n, causal)
    o2, l2 = torch.empty_like(o), torch.empty_like(l)
    fa.run_flash_bf16(handle, q, k, v, o2, l2, n, causal)
    handle.check_status()
    assert torch.equal(o, o2) and torch.equal(l, l2)
    for h in range(min(heads, 5)):
        s = q[h].double() @ k[h].double().T * 0.125
        if causal:
            s = s.masked_fill(torch.triu(torch.ones(n, n, dtype=torch.bool, device="cuda"), 1), -float("inf"))
        assert (o[h].double() - torch.softmax(s, -1) @ v[h].double()).abs().max() <= 2.2e-2
        assert (l[h].double() - torch.logsumexp(s, -1)).abs().max() <= (2e-3 if h % 3 == 1 else 1e-5)
        one, l_one = torch.empty(n, 64, device="cuda"), torch.empty(n, device="cuda")
        fa.run_flash_bf16(handle, q[h], k[h], v[h], one, l_one, n, causal)
        if h % 3 != 1:     # the max-free loop gives a head the same bits in either form of the kernel
            if n > 1920:
                assert torch.equal(one, o[h]) and torch.equal(l_one, l[h])


@pytest.mark.parametrize("heads", [2, 8, 40])   # 64-row, key-split, pair form
def test_bf16_forward_non_finite_operand(handle, heads):
    """A NaN in one head leaves the other heads alone and reaches every row of its own head that sees it."""
    n = 2048
    g = torch.Generator(device="cuda")
    g.manual_seed(6)
    q, k, v = (torch.randn(heads, n, 64, device="cuda", generator=g).bfloat16() for _ in range(3))
    o, l = torch.empty(heads, n, 64, device="cuda"), torch.empty(heads, n, device="cuda")
    fa.run_flash_bf16(handle, q, k, v, o, l, n, False)
    k[1, 777, 5] = float("nan")
    o2, l2 = torch.empty_like(o), torch.empty_like(l)
    fa.run_flash_bf16(handle, q, k, v, o2, l2, n, False)
    handle.check_status()
    others = [h for h in range(heads) if h != 1]
    assert torch.equal(o[others], o2[others]) and torch.equal(l[others], l2[others])
    assert torch.isnan(l2[1]).all()


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("heads,n", [(384, 64), (700, 128), (384, 300), (700, 300), (900, 129)])
def test_many_heads_with_an_odd_number_of_query_tiles(handle, heads, n, causal, bf16):
    """Pair form, several items per SM of which some or all have one query tile only, one after the other: the last rows of
    every head.  Against 64-bit softmax with the bounds of the test above; fp32 operands: q and k are rounded to bf16 as well,
    which moves a score by 1.6e-3 (sd; below 1.5e-2 over all of these), L by no more and a row by a quarter of twice that times
    the spread of v (below 11).  The sharp check for those: the same bits as the head in a call of its own."""
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    q, k, v = (torch.randn(heads, n, 64, device="cuda", generator=g) for _ in range(3))
    if bf16:
        q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    run = fa.run_flash_bf16 if bf16 else fa.run_flash_lse
    handle.reserve(fa.workspace_bytes(heads, n, False))
    o, l = torch.full((heads, n, 64), float("nan"), device="cuda"), torch.full((heads, n), float("nan"), device="cuda")
    run(handle, q, k, v, o, l, n, causal)
    handle.check_status()
    s = q.double() @ k.double().transpose(1, 2) * 0.125
    if causal:
        s = s.masked_fill(torch.triu(torch.ones(n, n, dtype=torch.bool, device="cuda"), 1), -float("inf"))
    assert (o.double() - torch.softmax(s, -1) @ v.double()).abs().max() <= (2.2e-2 if bf16 else 1e-1)
    assert (l.double() - torch.logsumexp(s, -1)).abs().max() <= (1e-5 if bf16 else 1.5e-2)
    if not bf16:
        one, l_one = torch.empty(n, 64, device="cuda"), torch.empty(n, device="cuda")
        for h in (0, 1, 147, 148, 295, 296, heads - 1):
            run(handle, q[h], k[h], v[h], one, l_one, n, causal)
            assert torch.equal(one, o[h]) and torch.equal(l_one, l[h]), f"head {h}"


@pytest.mark.parametrize("heads,n,causal", [(12, 2048, True), (14, 2177, True), (17, 2100, False)])   # key-split, over 148 items
@pytest.mark.parametrize("every,first", [(3, 1), (2, 0), (5, 2)])
def test_bf16_heads_inside_and_outside_the_bound_key_split(handle, heads, n, causal, every, first):
    """Several items per SM, an item of the general loop followed by one of the max-free loop, whose odd groups take their
    reference from the even ones' exchange: the bits of the head in a call of its own, and of every repetition."""
    g = torch.Generator(device="cuda")
    g.manual_seed(8)
    q, k, v = (torch.randn(heads, n, 64, device="cuda", generator=g) for _ in range(3))
    beyond = [h for h in range(heads) if h % every == first]
    q[beyond] *= 30
    q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    o, l = torch.empty(heads, n, 64, device="cuda"), torch.empty(heads, n, device="cuda")
    o2, l2 = torch.empty_like(o), torch.empty_like(l)
    fa.run_flash_bf16(handle, q, k, v, o, l, n, causal)
    for _ in range(10):
        fa.run_flash_bf16(handle, q, k, v, o2, l2, n, causal)
        assert torch.equal(o, o2) and torch.equal(l, l2)
    handle.check_status()
    for h in range(heads):
        s = q[h].double() @ k[h].double().T * 0.125
        if causal:
            s = s.masked_fill(torch.triu(torch.ones(n, n, dtype=torch.bool, device="cuda"), 1), -float("inf"))
        assert (o[h].double() - torch.softmax(s, -1) @ v[h].double()).abs().max() <= 2.2e-2   # as above
        if h not in beyond:
            one, l_one = torch.empty(n, 64, device="cuda"), torch.empty(n, device="cuda")
            fa.run_flash_bf16(handle, q[h], k[h], v[h], one, l_one, n, causal)
            assert torch.equal(one, o[h]) and torch.equal(l_one, l[h]), f"head {h}"
    handle.check_status()


@pytest.mark.parametrize("n", [1921, 4096, 5000])
@pytest.mark.parametrize("heads", [3, 8])   # 1921 rows: 64-row and key-split form
@pytest.mark.parametrize("where", ["first", "last", "apart", "swapped"])
def test_bf16_bound_is_of_the_whole_head(handle, n, heads, where):
    """One row of one operand decides the loop: the first or the last row of a head, of Q or of K, or large rows of Q against
    small ones of K that stay inside the bound.  The decision shows in L only by rounding, so the bound is the existing
    tests': the rows of 64-bit softmax, L to 2e-3 where scores reach 2^9."""
    g = torch.Generator(device="cuda")
    g.manual_seed(9)
    q, k, v = (torch.randn(heads, n, 64, device="cuda", generator=g) for _ in range(3))
    if where == "first":
        q[1, 0] *= 60
    elif where == "last":
        k[1, n - 1] *= 60
    elif where == "apart":
        q[0, 3] *= 10
        k[0, n - 2] *= 10
    else:
        q *= 64
        k /= 64
    q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    o, l = torch.empty(heads, n, 64, device="cuda"), torch.empty(heads, n, device="cuda")
    fa.run_flash_bf16(handle, q, k, v, o, l, n, False)
    handle.check_status()
    for h in range(heads):
        s = q[h].double() @ k[h].double().T * 0.125
        assert (o[h].double() - torch.softmax(s, -1) @ v[h].double()).abs().max() <= 2.2e-2
        assert (l[h].double() - torch.logsumexp(s, -1)).abs().max() <= 2e-3


@pytest.mark.parametrize("bf16,heads,n", [(False, 12, 2048), (False, 20, 1900), (True, 12, 1900), (True, 20, 1810)])
@pytest.mark.parametrize("every,first", [(3, 1), (2, 0), (5, 2)])
def test_odd_groups_publish_early_over_several_items(handle, bf16, heads, n, every, first):
    """Causal, key-split, 180 to 300 items: the odd groups hand on an item's sums before its last P V, item after item, over fp32
    operands (heads inside and beyond the bound) and bf16 ones without a bound.  The bits of every repetition and, in the max-free
    loop, of the head in a call of its own; else that call's rows to 2 * 2^-9 * max|v| (each takes P, rounded to bf16, against
    other maxima; max|v| < 5.5)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(10)
    q, k, v = (torch.randn(heads, n, 64, device="cuda", generator=g) for _ in range(3))
    beyond = [h for h in range(heads) if h % every == first]
    q[beyond] *= 30
    if bf16:
        q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    run = fa.run_flash_bf16 if bf16 else fa.run_flash_lse
    handle.reserve(fa.workspace_bytes(heads, n, False))
    o, l = torch.empty(heads, n, 64, device="cuda"), torch.empty(heads, n, device="cuda")
    o2, l2 = torch.empty_like(o), torch.empty_like(l)
    run(handle, q, k, v, o, l, n, True)
    for _ in range(10):
        run(handle, q, k, v, o2, l2, n, True)
        assert torch.equal(o, o2) and torch.equal(l, l2)
    one, l_one = torch.empty(n, 64, device="cuda"), torch.empty(n, device="cuda")
    for h in range(heads):
        run(handle, q[h], k[h], v[h], one, l_one, n, True)
        if not bf16 and h not in beyond:
            assert torch.equal(one, o[h]) and torch.equal(l_one, l[h]), f"head {h}"
        else:
            assert (one - o[h]).abs().max() <= 2.2e-2 and (l_one - l[h]).abs().max() <= 1e-3, f"head {h}"
    handle.check_status()

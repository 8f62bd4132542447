"""fp32 decode, the tile loop: every number of heads a CTA has code for (1, 2, 4, 7, 8 and those that fall to the next larger), the
last tile of every length, the shares of the warps, and how a tile finds its rows in a paged cache."""
import pytest
import torch

from mx230_b200 import llm_attention as la

pytestmark = pytest.mark.gpu


def attention64(row, k, v, nh, nkv, keys):
    q = row[:nh * 64].double().view(nh, 64)
    k, v = (x[:keys].double().view(keys, nkv, 64).repeat_interleave(nh // nkv, 1) for x in (k, v))
    return torch.einsum("ht,thd->hd", torch.softmax(torch.einsum("hd,thd->ht", q, k) * 0.125, -1), v).reshape(-1)


@pytest.mark.parametrize("nh,nkv", [(1, 1), (12, 12), (2, 1), (3, 1), (8, 2), (5, 1), (14, 2), (8, 1), (32, 4), (11, 1), (40, 20)])
def test_lengths_and_block_sizes(handle, nh, nkv):
    """Against 64 bits: scores of N(0,1) rows carry 2^-24 of about 8 standard deviations of partial sums, a row is an average of
    values of size 1: below 2e-6 of the result's norm at any length here (measured 1e-7 to 4e-7).  A paged cache whose tiles lie
    in one block each (16, 32), one whose tiles straddle blocks (8, 24) and a linear one hold the same rows and give the same bits."""
    g = torch.Generator(device="cuda")
    g.manual_seed(21)
    stride = (nh + 2 * nkv) * 64
    for keys in (1, 3, 4, 5, 15, 16, 17, 31, 33, 64, 65, 127, 129, 300, 777, 1100):
        lin = la.KvCache(keys, nkv)
        lin.k.normal_(generator=g), lin.v.normal_(generator=g)
        row = torch.randn(stride, device="cuda", generator=g)
        out, other = torch.full((nh * 64,), float("nan"), device="cuda"), torch.empty(nh * 64, device="cuda")
        la.attn_decode(handle, out, row, lin, keys - 1, nh, nkv, 64)
        want = attention64(row, lin.k, lin.v, nh, nkv, keys)
        assert (out.double() - want).norm() <= 2e-6 * want.norm(), keys
        for bs in (8, 16, 24, 32):
            n_log = -(-keys // bs)
            table = torch.randperm(n_log + 2, device="cuda", generator=g)[:n_log].to(torch.int32)
            c = la.KvCache((n_log + 2) * bs, nkv)
            c.k.fill_(float("nan")), c.v.fill_(float("nan"))   # rows that no key has
            at = torch.arange(keys, device="cuda")
            phys = table[at // bs].long() * bs + at % bs
            c.k[phys], c.v[phys] = lin.k, lin.v
            other.fill_(float("nan"))
            la.attn_decode(handle, other, row, c, keys - 1, nh, nkv, 64, la.Paging(table, bs))
            assert torch.equal(out, other), (keys, bs)
    handle.check_status()


@pytest.mark.parametrize("nh,nkv", [(1, 1), (2, 1), (4, 1), (14, 2), (8, 1)])
@pytest.mark.parametrize("pos", [0, 1, 16, 130])
def test_an_infinite_value_of_the_new_token_stays_in_its_dims(handle, nh, nkv, pos):
    """The step's own key is taken by one of a warp's key lanes: the others add nothing, not 0 times its V row."""
    g = torch.Generator(device="cuda")
    g.manual_seed(22)
    c = la.KvCache(pos + 1, nkv)
    c.k.normal_(generator=g), c.v.normal_(generator=g)
    row = torch.randn((nh + 2 * nkv) * 64, device="cuda", generator=g)
    row[(nh + nkv) * 64 + 5] = float("inf")
    out = torch.empty(nh * 64, device="cuda")
    la.decode_step(handle, out, row, c, pos, nh, nkv, 64, 1e6)
    handle.check_status()
    out = out.view(nh, 64)
    hit = torch.zeros(nh, 64, dtype=torch.bool, device="cuda")
    hit[:nh // nkv, 5] = True
    assert torch.isinf(out[hit]).all() and torch.isfinite(out[~hit]).all()


@pytest.mark.parametrize("bs", [8, 16, 24, 48])
@pytest.mark.parametrize("nh,nkv,n_seq", [(12, 12, 20), (16, 8, 30), (24, 8, 30), (14, 2, 70), (16, 2, 70), (32, 4, 40)])
def test_ranges_of_several_tiles(handle, nh, nkv, n_seq, bs):
    """A warp's range of none to nine tiles, in a batch whose groups leave a sequence one CTA or two: a tile's rows are looked up two
    tiles ahead.  Rows beyond a sequence's keys are NaN.  Bound as above."""
    g = torch.Generator(device="cuda")
    g.manual_seed(23)
    n_log = -(-560 // bs)
    keys = torch.tensor([(1 + 37 * i) % 560 + 1 for i in range(n_seq)], device="cuda")
    keys[0] = 560
    table = torch.randperm(n_seq * n_log, device="cuda", generator=g).to(torch.int32).reshape(n_seq, n_log)
    c = la.KvCache(n_seq * n_log * bs, nkv)
    c.k.fill_(float("nan")), c.v.fill_(float("nan"))
    rows = torch.randn(n_seq, (nh + 2 * nkv) * 64, device="cuda", generator=g)
    out = torch.full((n_seq, nh * 64), float("nan"), device="cuda")
    want = []
    for s in range(n_seq):
        n = int(keys[s])
        at = torch.arange(n, device="cuda")
        phys = table[s][at // bs].long() * bs + at % bs
        k, v = (torch.randn(n, nkv * 64, device="cuda", generator=g) for _ in range(2))
        c.k[phys], c.v[phys] = k, v
        want.append(attention64(rows[s], k, v, nh, nkv, n))
    la.attn_decode_batched(handle, out, rows, c, (keys - 1).to(torch.int32), n_seq, nh, nkv, 64, la.Paging(table, bs), rows.shape[1], nh * 64)
    handle.check_status()
    want = torch.stack(want)
    assert ((out.double() - want).norm(dim=1) <= 2e-6 * want.norm(dim=1)).all()

"""The decode step (one sequence: RoPE, KV write and attention in the attention kernel; a batch: all rows written, then
attention) against the separate entry points: the rotated row and the cache must be the same bits, and the attention row must
meet the oracle on that very cache (a batch: have the same bits as well).

Positions sit at the edges of the kernels' splits: tiles of 16 (fp32) and 32 (int8) keys, one pass of a CTA (64 / 256
keys), a cluster of eight CTAs, the point from which a second cluster joins in.  The tolerance of the row is that of the
decode tests (all arithmetic fp32, other summation order)."""
import numpy as np
import pytest
import torch

import oracle
from mx230_b200 import _lib
from mx230_b200 import llm_attention as la
from mx230_b200._lib import Mx230Error
from mx230_b200.common import Handle
from tests.conftest import assert_close

pytestmark = pytest.mark.gpu
TOL = dict(max_abs=2e-5, mean_rel=1e-4)
BS, THETA = 16, 1e6
HEADS = [(14, 2), (32, 4), (12, 12), (6, 2), (2, 1), (18, 1)]   # groups 7, 8, 1, 3, 2 and 18 (three launches)


def filled_cache(h, slots, nkv, quant, affine=True):
    g = torch.Generator(device="cuda")
    g.manual_seed(slots + nkv)
    c = la.KvCache(slots, nkv, 64, quant, affine)
    rows = torch.randn(slots, 2 * nkv * 64, device="cuda", generator=g)
    if quant:
        la.quantize_kv_batch(h, c, rows, 0, slots, 0, nkv, 64, 2 * nkv * 64)
    else:
        la.copy_kv_batch(h, c, rows, 0, slots, 0, nkv * 64, 2 * nkv * 64)
    return c


def copy_of(c):
    d = la.KvCache(c.slots, c.n_kv_head, 64, c.quant, c.affine)
    for n in ("k", "v") + (("ks", "vs") + (("kb", "vb") if c.affine else ()) if c.quant else ()):
        getattr(d, n).copy_(getattr(c, n))
    return d


def same_cache(a, b, what):
    for n in ("k", "v") + (("ks", "vs") + (("kb", "vb") if a.affine else ()) if a.quant else ()):
        assert torch.equal(getattr(a, n), getattr(b, n)), f"{what}: cache array {n} differs"


def oracle_rows(c, q, pos, nh, table):
    """The oracle's attention of one rotated row over the device's cache."""
    nkv = c.n_kv_head
    if c.quant:
        w = oracle.Q8Cache(c.slots, nkv, 64, c.affine)
        w.kq[:], w.vq[:], w.ks[:], w.vs[:] = (x.cpu().numpy() for x in (c.k, c.v, c.ks, c.vs))
        if c.affine:
            w.kb[:], w.vb[:] = c.kb.cpu().numpy(), c.vb.cpu().numpy()
        return oracle.gqa_decode_q8(q, w, pos, nh, 1, table, BS)
    return oracle.gqa_decode_f32(q, c.k.cpu().numpy(), c.v.cpu().numpy(), pos, nh, nkv, 64, table, BS)


@pytest.mark.parametrize("quant,affine", [(False, True), (True, True), (True, False)])
@pytest.mark.parametrize("nh,nkv", HEADS)
@pytest.mark.parametrize("paged", [False, True])
def test_single_sequence_step(handle, nh, nkv, quant, affine, paged):
    qd, kvd = nh * 64, nkv * 64
    slots = 4608
    c0 = filled_cache(handle, slots, nkv, quant, affine)
    table = np.random.default_rng(3).permutation(slots // BS).astype(np.int32) if paged else None
    pg = la.Paging(torch.from_numpy(table).cuda(), BS) if paged else None
    for pos in (0, 1, 15, 16, 63, 64, 65, 255, 256, 511, 1023, 2047, 2049, 4095, 4097, 4607):
        raw = torch.from_numpy(oracle.normal((qd + 2 * kvd,), 900 + pos, nh)).cuda()
        sep, fused, dyn = raw.clone(), raw.clone(), raw.clone()
        cs, cf, cd = copy_of(c0), copy_of(c0), copy_of(c0)
        row = pg.phys_row(table, pos) if paged else pos
        la.rope(handle, sep, pos, nh, nkv, 64, THETA)
        if quant:
            la.quantize_kv(handle, cs, sep, row, qd, nkv, 64)
        else:
            la.copy_kv(handle, cs, sep, row, qd, kvd)
        out = torch.full((qd,), float("nan"), device="cuda")
        la.decode_step(handle, out, fused, cf, pos, nh, nkv, 64, THETA, pg, table)
        out_dyn = torch.full((qd,), float("nan"), device="cuda")
        la.decode_step_dyn(handle, out_dyn, dyn, cd, torch.tensor([pos], dtype=torch.int32, device="cuda"), nh, nkv, 64, THETA, pg)
        assert torch.equal(fused, sep) and torch.equal(dyn, sep), f"pos {pos}: rotated row"
        same_cache(cf, cs, f"pos {pos}")
        same_cache(cd, cs, f"pos {pos} dyn")
        want = oracle_rows(cs, sep.cpu().numpy(), pos, nh, table)
        assert_close(out.cpu().numpy(), want, f"pos {pos}", **TOL)
        assert_close(out_dyn.cpu().numpy(), want, f"pos {pos} dyn", **TOL)
    handle.check_status()


@pytest.mark.parametrize("quant", [False, True])
@pytest.mark.parametrize("nh,nkv,n_seq,ctx", [(14, 2, 3, 700), (14, 2, 20, 600), (14, 2, 80, 300), (32, 4, 37, 500), (12, 12, 5, 1100),
                                              (18, 1, 4, 90), (14, 2, 150, 40)])
def test_batched_step(handle, nh, nkv, n_seq, ctx, quant):
    qd, kvd = nh * 64, nkv * 64
    stride, out_stride = qd + 2 * kvd + 64, qd + 32
    n_log = -(-ctx // BS)
    rng = np.random.default_rng(n_seq + ctx)
    pos = rng.integers(0, ctx, n_seq).astype(np.int32)
    pos[0], pos[-1] = ctx - 1, 0
    tables = rng.permutation(n_seq * n_log).astype(np.int32).reshape(n_seq, n_log)
    pg = la.Paging(torch.from_numpy(tables).cuda(), BS)
    cs = filled_cache(handle, n_seq * n_log * BS, nkv, quant)
    cf = copy_of(cs)
    posd = torch.from_numpy(pos).cuda()
    raw = torch.from_numpy(oracle.normal((n_seq, stride), 77, n_seq)).cuda()
    sep, fused = raw.clone(), raw.clone()
    la.rope_seqpos(handle, sep, posd, n_seq, nh, nkv, 64, stride, THETA)
    if quant:
        la.quantize_kv_seqpos(handle, cs, sep, posd, n_seq, qd, nkv, 64, stride, pg)
    else:
        la.copy_kv_seqpos(handle, cs, sep, posd, n_seq, qd, kvd, stride, pg)
    out = torch.zeros(n_seq, out_stride, device="cuda")
    la.batched_step(handle, out, fused, cf, posd, n_seq, nh, nkv, 64, THETA, pg, stride, out_stride)
    out_sep = torch.zeros_like(out)
    la.attn_decode_batched(handle, out_sep, sep, cs, posd, n_seq, nh, nkv, 64, pg, stride, out_stride)
    assert torch.equal(fused, sep) and torch.equal(out, out_sep)
    same_cache(cf, cs, "batched step")
    got, rows = out.cpu().numpy(), sep.cpu().numpy()
    assert (got[:, qd:] == 0).all()   # padding of the output rows is not touched
    for i in sorted({0, 1, n_seq // 2, n_seq - 1}):
        want = oracle_rows(cs, np.ascontiguousarray(rows[i]), int(pos[i]), nh, tables[i])
        assert_close(got[i, :qd], want, f"sequence {i} at {pos[i]}", **TOL)
    handle.check_status()


@pytest.mark.parametrize("quant,affine", [(False, True), (True, True), (True, False)])
@pytest.mark.parametrize("nh,nkv", [(14, 2), (12, 12), (18, 1)])
@pytest.mark.parametrize("rows,first", [(2, 0), (5, 30), (16, 500), (40, 1000)])
def test_rows_of_one_sequence(handle, nh, nkv, quant, affine, rows, first):
    """Consecutive positions of one sequence as rows of one batched step (a draft's verification, a chunk through the decode
    path), beside a sequence that shares its first blocks: each row sees the keys that the call itself writes."""
    qd, kvd = nh * 64, nkv * 64
    stride = qd + 2 * kvd
    n_log = (first + rows) // BS + 2
    rng = np.random.default_rng(rows)
    table = rng.permutation(2 * n_log).astype(np.int32)
    other = table[n_log:].copy()
    other[:first // BS] = table[:first // BS]
    tables = np.concatenate([np.tile(table[:n_log], (rows, 1)), other[None]])
    pos = np.concatenate([first + rng.permutation(rows), [first]]).astype(np.int32)
    n_seq = rows + 1
    pg, posd = la.Paging(torch.from_numpy(tables).cuda(), BS), torch.from_numpy(pos).cuda()
    c0 = filled_cache(handle, 2 * n_log * BS, nkv, quant, affine)
    raw = torch.from_numpy(oracle.normal((n_seq, stride), 78, rows)).cuda()
    sep, cs = raw.clone(), copy_of(c0)
    la.rope_seqpos(handle, sep, posd, n_seq, nh, nkv, 64, stride, THETA)
    if quant:
        la.quantize_kv_seqpos(handle, cs, sep, posd, n_seq, qd, nkv, 64, stride, pg)
    else:
        la.copy_kv_seqpos(handle, cs, sep, posd, n_seq, qd, kvd, stride, pg)
    want = torch.empty(n_seq, qd, device="cuda")
    la.attn_decode_batched(handle, want, sep, cs, posd, n_seq, nh, nkv, 64, pg, stride, qd)
    for _ in range(5):
        step, c, out = raw.clone(), copy_of(c0), torch.empty(n_seq, qd, device="cuda")
        la.batched_step(handle, out, step, c, posd, n_seq, nh, nkv, 64, THETA, pg, stride, qd)
        assert torch.equal(step, sep) and torch.equal(out, want)
        same_cache(c, cs, "rows of one sequence")
    for i in (0, rows - 1, rows):
        w = oracle_rows(cs, np.ascontiguousarray(sep[i].cpu().numpy()), int(pos[i]), nh, tables[i])
        assert_close(out[i].cpu().numpy(), w, f"row {i} at {pos[i]}", **TOL)
    handle.check_status()


@pytest.mark.parametrize("quant", [False, True])
@pytest.mark.parametrize("nh,nkv", [(14, 2), (18, 1)])
def test_device_position_must_be_given(handle, nh, nkv, quant):
    """A null device position is refused, and row and cache are left alone."""
    c = filled_cache(handle, 64, nkv, quant)
    before, qkv = copy_of(c), torch.randn((nh + 2 * nkv) * 64, device="cuda")
    row, out = qkv.clone(), torch.zeros(nh * 64, device="cuda")
    with pytest.raises(Mx230Error):
        la.decode_step_dyn(handle, out, qkv, c, None, nh, nkv, 64, THETA)
    assert torch.equal(qkv, row) and (out == 0).all()
    same_cache(c, before, "refused step")


@pytest.mark.parametrize("quant", [False, True])
@pytest.mark.parametrize("nh,nkv", [(14, 2), (12, 12), (32, 4)])
@pytest.mark.parametrize("pos", [0, 40, 700, 4500])
def test_step_in_place(handle, nh, nkv, quant, pos):
    """out may be the qkv row itself, as with the separate calls: the attention row replaces q, K is left rotated."""
    qd = nh * 64
    c0 = filled_cache(handle, 4608, nkv, quant)
    raw = torch.from_numpy(oracle.normal((qd + 2 * nkv * 64,), 79, pos)).cuda()
    apart, inplace, ca, ci = raw.clone(), raw.clone(), copy_of(c0), copy_of(c0)
    out = torch.empty(qd, device="cuda")
    la.decode_step(handle, out, apart, ca, pos, nh, nkv, 64, THETA)
    la.decode_step(handle, inplace, inplace, ci, pos, nh, nkv, 64, THETA)
    assert torch.equal(inplace[:qd], out) and torch.equal(inplace[qd:], apart[qd:])
    same_cache(ca, ci, "step in place")
    handle.check_status()


@pytest.mark.parametrize("mode,nh,nkv,n_seq,ctx", [
    ("tensor", 14, 2, 64, 2048), ("exact", 14, 2, 64, 2048), ("exact", 14, 2, 60, 512), ("cores", 12, 12, 12, 4096),
    ("fp32", 14, 2, 80, 800),   # groups for four fifths of the SMs and room for two splits
])
def test_short_contexts_need_no_workspace(handle, mode, nh, nkv, n_seq, ctx):
    """A handle whose workspace holds no second split takes the call with one, and agrees with one that splits."""
    quant, qd = mode != "fp32", nh * 64
    n_log = ctx // BS
    rng = np.random.default_rng(ctx)
    c = filled_cache(handle, n_seq * n_log * BS, nkv, quant)
    pg = la.Paging(torch.from_numpy(rng.permutation(n_seq * n_log).astype(np.int32).reshape(n_seq, n_log)).cuda(), BS)
    pos = torch.from_numpy(np.concatenate([[ctx - 1, 0], rng.integers(0, ctx, n_seq - 2)]).astype(np.int32)).cuda()
    qkv = torch.from_numpy(oracle.normal((n_seq, qd + 2 * nkv * 64), 80, n_seq)).cuda()
    small = Handle(0, 4096)
    rows = []
    try:
        for h in (small, handle):
            h.set_option(_lib.OPT_Q8_SCORE_MODE, _lib.Q8_SCORE_EXACT if mode == "exact" else _lib.Q8_SCORE_REF)
            h.set_option(_lib.OPT_DECODE_TENSOR, int(mode != "cores"))
            rows.append(torch.empty(n_seq, qd, device="cuda"))
            la.attn_decode_batched(h, rows[-1], qkv, c, pos, n_seq, nh, nkv, 64, pg, qkv.shape[1], qd)
            h.check_status()
    finally:
        handle.set_option(_lib.OPT_Q8_SCORE_MODE, _lib.Q8_SCORE_REF)
        handle.set_option(_lib.OPT_DECODE_TENSOR, 1)
        small.close()
    assert_close(rows[0].cpu().numpy(), rows[1].cpu().numpy(), mode, **TOL)

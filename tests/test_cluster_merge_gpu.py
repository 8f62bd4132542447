"""The cluster merge of decode attention and of the projections when CTAs wait for one another longer than they may: with the
smallest bound that a handle takes an ordinary call is still right and leaves no status, for only stores that are issued are
waited for against the bound.  Where sums never come (a test hook) the launch ends with a status and the handle keeps working."""
import numpy as np
import pytest
import torch

import oracle
from mx230_b200 import _lib
from mx230_b200 import llm_attention as la
from mx230_b200.common import Handle
from tests.conftest import assert_close
from tests.test_decode_gpu import TOL, build_caches, dev, to_dev_f32, to_dev_q8
from tests.test_decode_step_gpu import filled_cache

pytestmark = pytest.mark.gpu


@pytest.fixture()
def own_handle(lib_built):
    torch.cuda.set_device(0)
    h = Handle(0, 64 << 20)
    yield h
    h.close()


@pytest.mark.parametrize("nh,nkv", [(7, 1), (14, 2), (12, 12)])
def test_decode_with_the_smallest_bound(own_handle, nh, nkv):
    h = own_handle
    rows, kc, vc, q8 = build_caches(nh, nkv, 4500, 43)
    c32, c8 = to_dev_f32(kc, vc, nkv), to_dev_q8(q8)
    out = torch.empty(nh * 64, device="cuda")
    h.set_option(_lib.OPT_WAIT_LIMIT, 1)
    for t in (129, 1024, 4499):   # known to the host: a cluster of two or three, one of up to eight, several CTAs or clusters
        pos = torch.tensor([t], dtype=torch.int32, device="cuda")
        w32, w8 = oracle.gqa_decode_f32(rows[t], kc, vc, t, nh, nkv), oracle.gqa_decode_q8(rows[t], q8, t, nh, 1)
        for _ in range(20):
            for c, want in ((c32, w32), (c8, w8)):
                for at, call in ((t, la.attn_decode), (pos, la.attn_decode_dyn)):
                    out.fill_(float("nan"))
                    call(h, out, dev(rows[t]), c, at, nh, nkv, 64)
                    h.check_status()
                    assert_close(out.cpu().numpy(), want, f"{t} keys", **TOL)


def test_projection_with_the_smallest_bound(own_handle):
    h = own_handle
    for n_in, n_out in ((896, 1152), (200, 132)):   # 38 slices in eight CTAs, 13 in seven, the last one short
        x, b = oracle.normal((n_in,), 51, 0), oracle.normal((n_out,), 51, 1)
        w = (oracle.normal((n_in, n_out), 51, 2) * 0.05).astype(np.float16)
        y = torch.empty(n_out, device="cuda")
        h.set_option(_lib.OPT_WAIT_LIMIT, 1)
        for _ in range(20):
            y.fill_(float("nan"))
            la.gemv(h, y, dev(x), dev(w), dev(b))
            h.check_status()
            assert_close(y.cpu().numpy(), oracle.gemv(x, w, b), "gemv", max_abs=2e-4, mean_rel=2e-5)


def _run_out(h, call):
    """The call with CTA 1 of its first cluster waiting for sums that nobody sends, and a bound of about a millisecond."""
    try:
        h.set_option(_lib.OPT_WAIT_LIMIT, 2000)
        h.set_option(_lib.OPT_TEST_DROP_TILE, 1)
        call()
        with pytest.raises(_lib.Mx230Error) as e:
            h.check_status()
        assert e.value.code == _lib.ERR_DEVICE_STATUS
    finally:
        h.set_option(_lib.OPT_TEST_DROP_TILE, -1)
        h.set_option(_lib.OPT_WAIT_LIMIT, 4000000)


@pytest.mark.parametrize("quant", [False, True])
@pytest.mark.parametrize("keys", [600, 9000])   # one cluster, two: their partial rows go through the workspace
def test_decode_merge_that_runs_out(own_handle, quant, keys):
    """No row of an earlier call, which the workspace still holds, passes for one of the call that failed."""
    h, (nh, nkv) = own_handle, (14, 2)
    c = filled_cache(h, keys, nkv, quant)
    qkv = torch.randn(2, (nh + 2 * nkv) * 64, device="cuda")
    pos = torch.tensor([keys - 1], dtype=torch.int32, device="cuda")
    out = torch.zeros(nh * 64, device="cuda")

    def call(i):
        la.attn_decode_dyn(h, out, qkv[i], c, pos, nh, nkv, 64)
    call(0)
    h.check_status()
    want = out.clone()
    call(1)   # leaves its partial rows in the workspace
    _run_out(h, lambda: call(0))
    assert torch.isnan(out[64:128]).all()   # CTA 1 of eight finishes head 1
    assert torch.equal(out[:64], want[:64]) and torch.equal(out[128:], want[128:])
    call(0)
    h.check_status()
    assert torch.equal(out, want)


def test_projection_merge_that_runs_out(own_handle):
    h = own_handle
    x, w, b = torch.randn(896, device="cuda"), torch.randn(896, 1152, device="cuda").half(), torch.randn(1152, device="cuda")
    y = torch.zeros(1152, device="cuda")
    la.gemv(h, y, x, w, b)
    h.check_status()
    want = y.clone()
    y.fill_(7.0)
    _run_out(h, lambda: la.gemv(h, y, x, w, b))
    assert (y[:64] == 7.0).all() and torch.equal(y[64:], want[64:])
    la.gemv(h, y, x, w, b)
    h.check_status()
    assert torch.equal(y, want)

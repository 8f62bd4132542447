"""The cluster merge of decode attention and of the projections when CTAs wait for one another longer than they may: with the
smallest bound that a handle takes an ordinary call is still right and leaves no status, for only stores that are issued are
waited for against the bound."""
import numpy as np
import pytest
import torch

import oracle
from mx230_b200 import _lib
from mx230_b200 import llm_attention as la
from mx230_b200.common import Handle
from tests.conftest import assert_close
from tests.test_decode_gpu import TOL, build_caches, dev, to_dev_f32, to_dev_q8

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

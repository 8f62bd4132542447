"""Decode attention merged over thread-block clusters of every size: one sequence, whose number of keys sets the cluster (a CTA
for every 64 or 128 fp32 or 256 int8 keys, up to eight), and every way the heads of a group can fall to the cluster's CTAs."""
import pytest
import torch

import oracle
from mx230_b200 import llm_attention as la
from mx230_b200.common import Handle
from tests.conftest import assert_close
from tests.test_decode_gpu import TOL, build_caches, dev, to_dev_f32, to_dev_q8

pytestmark = pytest.mark.gpu


# groups of 7, 8, 3, 5, 1 heads; with 20 K/V heads the fp32 CTAs have four warps, in the other calls eight
@pytest.mark.parametrize("nh,nkv", [(7, 1), (8, 1), (3, 1), (10, 2), (5, 5), (20, 20)])
def test_every_cluster_size(handle, nh, nkv):
    rows, kc, vc, q8 = build_caches(nh, nkv, 2049, 41)
    c32, c8 = to_dev_f32(kc, vc, nkv), to_dev_q8(q8)
    out = torch.empty(nh * 64, device="cuda")
    for size in range(1, 9):
        for keys in {64 * size, 64 * size + 1, 128 * size, 128 * size + 1}:
            row = rows[keys - 1]
            out.fill_(float("nan"))
            la.attn_decode(handle, out, dev(row), c32, keys - 1, nh, nkv, 64)
            assert_close(out.cpu().numpy(), oracle.gqa_decode_f32(row, kc, vc, keys - 1, nh, nkv), f"fp32 {keys} keys", **TOL)
        for keys in {256 * size - 255, 256 * size}:
            row = rows[keys - 1]
            out.fill_(float("nan"))
            la.attn_decode(handle, out, dev(row), c8, keys - 1, nh, nkv, 64)
            assert_close(out.cpu().numpy(), oracle.gqa_decode_q8(row, q8, keys - 1, nh, 1), f"int8 {keys} keys", **TOL)
    handle.check_status()


@pytest.mark.parametrize("nkv", [16, 17, 18])
def test_many_groups_with_little_workspace(lib_built, nkv):
    """Groups of which eight eight-warp CTAs each are not resident at once: up to two clusters of four-warp CTAs where the host
    knows the length, and one, without workspace, where the handle has none for more."""
    keys = 4096
    rows, kc, vc, _ = build_caches(nkv, nkv, keys, 44)
    c, row = to_dev_f32(kc, vc, nkv), rows[keys - 1]
    want = oracle.gqa_decode_f32(row, kc, vc, keys - 1, nkv, nkv)
    pos = torch.tensor([keys - 1], dtype=torch.int32, device="cuda")
    for splits in (2, 0):
        h = Handle(0, nkv * 66 * 4 * splits)
        for at, call in ((keys - 1, la.attn_decode), (pos, la.attn_decode_dyn)):
            out = torch.full((nkv * 64,), float("nan"), device="cuda")
            call(h, out, dev(row), c, at, nkv, nkv, 64)
            h.check_status()
            assert_close(out.cpu().numpy(), want, f"{splits} {call.__name__}", **TOL)
        h.close()

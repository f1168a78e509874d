"""GPU: grouped-query backward whose query-head group is split over several CTAs (fp32 partial dK / dV, summed in a
fixed order), against the oracle: uneven parts, ragged last tiles, both dQ modes."""
import ctypes

import pytest
import torch

from oracle import dense_oracle as orc
from tests.util import assert_close, bernoulli_mask, rand_qkv

pytestmark = pytest.mark.gpu

CASES = {
    # name: (B, Hq, Hkv, Sq, Skv, qb, kb, keep)
    "group_2": (1, 2, 1, 512, 384, 128, 128, 0.5),
    "group_3": (2, 6, 2, 384, 640, 128, 128, 0.5),
    "group_5": (1, 5, 1, 768, 1280, 128, 128, 0.3),
    "multi_query_24": (1, 24, 1, 384, 1280, 384, 128, 0.4),
    "ragged": (2, 8, 2, 336, 576, 48, 192, 0.5),
    "sparse_empty_lists": (1, 4, 1, 640, 640, 128, 128, 0.1),
}


@pytest.mark.parametrize("mode", ["atomic", "qmajor"])
@pytest.mark.parametrize("name", list(CASES))
def test_split_groups(name, mode):
    import flex_block_attn_b200 as fba
    from flex_block_attn_b200 import _cabi

    B, Hq, Hkv, Sq, Skv, qb, kb, keep = CASES[name]
    n = ctypes.c_uint64(0)
    assert _cabi.lib().fba_bwd_partial_bytes(B, Hq, Hkv, Sq, Skv, ctypes.byref(n)) == 0
    assert n.value > 0, "these sizes are meant to be split"
    q, k, v, do = rand_qkv(B, Hq, Hkv, Sq, Skv, seed=11, device="cuda")
    mask = bernoulli_mask((B, Hq, Sq // qb, Skv // kb), keep, 11, force_diag=False).cuda()
    lists = fba.build_lists(mask, qb, kb, Sq, Skv)
    o, lse = fba.forward_with_lists(q, k, v, lists)
    got = fba.backward_with_lists(q, k, v, o, lse, do, lists, dq_mode=mode)
    again = fba.backward_with_lists(q, k, v, o, lse, do, lists, dq_mode=mode)
    torch.cuda.synchronize()
    fba.check_status()
    assert torch.equal(got[1], again[1]) and torch.equal(got[2], again[2]), "dK / dV must be reproducible"
    want = orc.attention_slab(q.float(), k.float(), v.float(), mask, qb, kb, do.float())
    for a, w, nm in zip(got, want[2:], ("dQ", "dK", "dV")):
        assert_close(a.float(), w, f"{name} {mode} {nm}")

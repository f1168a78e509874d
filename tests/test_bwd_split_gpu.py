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


PARTLY_FILLED = {
    # name: (B, Hq, Hkv, Sq, Skv, qb, kb, mask dims, split key tiles, parts); one wave is 148 key tiles
    "whole_wave_and_4": (2, 8, 2, 336, 4800, 48, 192, 4, 4, 4),
    "whole_wave_and_2_shared_mask": (1, 6, 1, 512, 19200, 128, 128, 2, 2, 6),
    "two_waves_and_12": (2, 10, 2, 256, 9856, 128, 128, 4, 12, 5),
    "uneven_parts": (1, 5, 1, 384, 6400, 384, 128, 4, 50, 2),
    "largest_split_tail": (1, 2, 1, 256, 9472, 128, 128, 4, 74, 2),
    "tail_too_large": (1, 2, 1, 256, 9600, 128, 128, 4, 0, 1),
    "no_tail": (1, 2, 1, 256, 18944, 128, 128, 4, 0, 1),
}


@pytest.mark.parametrize("name", list(PARTLY_FILLED))
def test_split_of_a_partly_filled_wave(name, monkeypatch):
    """As many tiles are split as a partly filled wave would have; the others have the unsplit call's bits, and neither
    the work order nor the dQ mode changes any of dK and dV."""
    import flex_block_attn_b200 as fba
    from flex_block_attn_b200 import _cabi

    B, Hq, Hkv, Sq, Skv, qb, kb, dims, tail, parts = PARTLY_FILLED[name]
    lib, n, n1, n2 = _cabi.lib(), ctypes.c_uint64(0), ctypes.c_uint64(0), ctypes.c_uint64(0)
    assert lib.fba_bwd_partial_bytes(B, Hq, Hkv, Sq, Skv, ctypes.byref(n)) == 0
    assert n.value == (tail * parts * 2 * 65536 if parts > 1 else 0)
    q, k, v, do = rand_qkv(B, Hq, Hkv, Sq, Skv, seed=21, device="cuda")
    shape = (Sq // qb, Skv // kb) if dims == 2 else (B, Hq, Sq // qb, Skv // kb)
    mask = bernoulli_mask(shape, 0.4, 21, force_diag=False).cuda()
    runs = []
    for order, mode in (("1", "atomic"), ("0", "atomic"), ("1", "qmajor")):
        monkeypatch.setenv("FBA_WORK_ORDER", order)
        lists = fba.build_lists(mask, qb, kb, Sq, Skv)
        o, lse = fba.forward_with_lists(q, k, v, lists)
        runs.append(fba.backward_with_lists(q, k, v, o, lse, do, lists, dq_mode=mode))
    for r in runs[1:]:
        assert torch.equal(r[1], runs[0][1]) and torch.equal(r[2], runs[0][2])
    want = orc.attention_slab(q.float(), k.float(), v.float(), mask, qb, kb, do.float())
    for a, w, nm in zip(runs[0], want[2:], ("dQ", "dK", "dV")):
        assert_close(a.float(), w, f"{name} {nm}")
    # the same lists without a partial buffer, and with one that is not touched beside its stated size
    assert lib.fba_bwd_scratch_bytes(B, Hq, Sq, ctypes.byref(n1), ctypes.byref(n2)) == 0
    ld, acc = torch.empty(n1.value // 4, device="cuda"), torch.empty(n2.value // 4, device="cuda")
    room = torch.full((n.value // 4 + 64,), 77.0, device="cuda")
    lst = lists.bwd_list(Hq, Hkv)
    stream, status = torch.cuda.current_stream().cuda_stream, fba.interface._status(q.device).data_ptr()
    res = []
    for partial in (None, room.data_ptr()):
        g = [torch.full_like(x, float("nan")) for x in (q, k, v)]
        ptrs = [x.data_ptr() for x in (q, k, v, o, lse, do, *g)]
        _cabi.check(lib.fba_bwd_split(*ptrs, B, Hq, Hkv, Sq, Skv, ctypes.byref(lst), None, 128 ** -0.5, 0, ld.data_ptr(),
                                      acc.data_ptr(), partial, n.value, status, stream), "fba_bwd_split")
        res.append(g)
    torch.cuda.synchronize()
    fba.check_status()
    assert (room[n.value // 4:] == 77.0).all()
    n_tiles = B * Hkv * -(-Skv // 128)
    whole = torch.arange(n_tiles, device="cuda").view(B, Hkv, -1) < n_tiles - tail
    rows = whole.repeat_interleave(128, -1)[..., :Skv]
    for i, nm in ((1, "dK"), (2, "dV")):
        assert torch.equal(res[1][i], runs[0][i])
        assert torch.equal(res[0][i][rows], runs[0][i][rows]), f"{nm} of an unsplit tile"
        assert_close(res[0][i].float(), want[2 + i], f"{name} unsplit {nm}")


def test_attn_backward_workspace_without_room_for_the_split():
    """fba_attn_backward with the reported workspace splits like the list-level call; without the last part of it, or a
    byte short, it runs unsplit: the bits of fba_bwd_ex."""
    import flex_block_attn_b200 as fba
    from flex_block_attn_b200 import _cabi

    lib = _cabi.lib()
    B, Hq, Hkv, S, blk = 1, 4, 1, 1536, 128
    q, k, v, do = rand_qkv(B, Hq, Hkv, S, S, seed=31, device="cuda")
    mask = bernoulli_mask((B, Hq, S // blk, S // blk), 0.5, 31).cuda()
    lists = fba.build_lists(mask, blk, blk, S, S)
    o, lse = fba.forward_with_lists(q, k, v, lists)
    split = fba.backward_with_lists(q, k, v, o, lse, do, lists)
    stream, status = torch.cuda.current_stream().cuda_stream, fba.interface._status(q.device).data_ptr()
    n, part, n1, n2 = (ctypes.c_uint64(0) for _ in range(4))
    assert lib.fba_attn_workspace_bytes(B, Hq, Hkv, S, S, blk, blk, 4, 1, ctypes.byref(n)) == 0
    assert lib.fba_bwd_partial_bytes(B, Hq, Hkv, S, S, ctypes.byref(part)) == 0 and part.value > 0
    assert lib.fba_bwd_scratch_bytes(B, Hq, S, ctypes.byref(n1), ctypes.byref(n2)) == 0
    ld, acc = torch.empty(n1.value // 4, device="cuda"), torch.empty(n2.value // 4, device="cuda")
    lst = lists.bwd_list(Hq, Hkv)

    def grads():
        g = [torch.full_like(x, float("nan")) for x in (q, k, v)]
        return g, [x.data_ptr() for x in (q, k, v, o, lse, do, *g)]

    whole, ptrs = grads()
    _cabi.check(lib.fba_bwd_ex(*ptrs, B, Hq, Hkv, S, S, ctypes.byref(lst), None, 128 ** -0.5, 0, ld.data_ptr(),
                               acc.data_ptr(), status, stream), "fba_bwd_ex")
    mask_t = mask.transpose(-1, -2).contiguous().view(torch.uint8)
    for size, want in ((n.value, split), (n.value - 1, whole), (n.value - (part.value + 255) // 256 * 256, whole)):
        ws = torch.full((size + 256,), 77, dtype=torch.uint8, device="cuda")
        assert ws.data_ptr() % 256 == 0
        got, ptrs = grads()
        _cabi.check(lib.fba_attn_backward(*ptrs, B, Hq, Hkv, S, S, blk, blk, mask_t.data_ptr(), None, 4, 0, ws.data_ptr(), size,
                                          status, stream), "fba_attn_backward")
        torch.cuda.synchronize()
        fba.check_status()
        assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
        assert_close(got[0].float(), want[0].float(), f"dQ, workspace of {size} bytes", max_abs=1e-2)
        assert (ws[size:] == 77).all()
    assert not torch.equal(split[1], whole[1])   # else the comparison above shows nothing

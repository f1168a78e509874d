"""GPU: the forward's two query tiles of a CTA take turns on one score buffer; lists of unequal length, empty
lists, a lone last tile and lists of one entry are where that hand-over can go wrong."""
import pytest
import torch

from oracle import dense_oracle as orc
from tests.util import assert_close, rand_qkv

pytestmark = pytest.mark.gpu

# entries of the list of each 128-row query tile; tiles 2p and 2p + 1 share a CTA
COUNTS = {
    "one_empty": (0, 5, 5, 0),
    "both_empty": (0, 0, 3, 3),
    "short_long": (1, 9, 9, 1),
    "off_by_one": (4, 5, 5, 4),
    "single_entries": (1, 1, 2, 1),
    "lone_last_tile": (9, 2, 7),
    "lone_tile": (6,),
}


@pytest.mark.parametrize("name", list(COUNTS))
def test_unequal_lists(name):
    import flex_block_attn_b200 as fba

    counts, nK = COUNTS[name], 9
    Sq, Skv = 128 * len(counts), 128 * nK
    q, k, v, do = rand_qkv(1, 2, 1, Sq, Skv, seed=7, device="cuda")
    g = torch.Generator().manual_seed(3)
    mask = torch.zeros((1, 2, len(counts), nK), dtype=torch.bool)
    for h in range(2):
        for r, n in enumerate(counts):
            mask[0, h, r, torch.randperm(nK, generator=g)[:n]] = True
    mask = mask.cuda()
    lists = fba.build_lists(mask, 128, 128, Sq, Skv, need_bwd=False)
    o, lse = fba.forward_with_lists(q, k, v, lists)
    torch.cuda.synchronize()
    fba.check_status()
    want = orc.attention_slab(q.float(), k.float(), v.float(), mask, 128, 128, do.float())
    # P and O are rounded to bf16 (2^-9 each); rows of a few keys reach |O| of about 4
    assert_close(o.float(), want[0], f"{name} O")
    dead = ~mask.any(-1).repeat_interleave(128, -1)
    assert torch.equal(o[dead], torch.zeros_like(o[dead]))
    assert torch.isneginf(lse[dead]).all() and torch.isfinite(lse[~dead]).all()

"""compact_plan's device pairing and list builder against the rule in plain torch and the oracle's lists, bit for bit."""
import pytest
import torch

import paroatten_b200 as pb
from oracle import paro_oracle as po
from paroatten_b200.plan import pair_rows_by_overlap

pytestmark = pytest.mark.gpu


def bernoulli(S, nbq, nbk, density):
    return torch.rand(S, nbq, nbk, generator=torch.Generator().manual_seed(nbq * 7 + nbk)) < density


def twins(nb):
    """q-block r of an even group of 32 keeps what q-block r+32 keeps, so whole groups of rows are used up as partners."""
    m = torch.zeros(1, nb, nb, dtype=torch.bool)
    r = torch.arange(nb)
    m[0, r, (r % 32) + 32 * (r // 64)] = True
    m[0, :, 0] = True
    return m


@pytest.mark.parametrize("mask", [
    bernoulli(3, 4, 4, 0.5), bernoulli(2, 5, 9, 0.5), bernoulli(2, 31, 33, 0.3), bernoulli(5, 64, 64, 0.2),
    bernoulli(2, 65, 1025, 0.1), bernoulli(1, 130, 2100, 0.6), bernoulli(2, 277, 278, 0.3), bernoulli(2, 40, 40, 0.0),
    bernoulli(2, 33, 33, 1.0), twins(193), twins(256)], ids=lambda m: "x".join(map(str, m.shape)))
def test_pairing_and_lists(mask):
    plan = pb.compact_plan(mask.cuda(), pairing="overlap", validate=bool(mask.any()))
    S, nbq, nbk = mask.shape
    order = pair_rows_by_overlap(mask.to(torch.uint8))
    tiles = lambda m: (m[:, 0::2][:, :nbq // 2] | m[:, 1::2]).sum(dim=(1, 2))
    rows = torch.gather(mask, 1, order.unsqueeze(-1).expand(-1, -1, nbk))
    better = tiles(rows) < tiles(mask)
    order = torch.where(better.unsqueeze(1), order, torch.arange(nbq).expand_as(order))
    rows = torch.gather(mask, 1, order.unsqueeze(-1).expand(-1, -1, nbk))
    ptr, cols = po.compact_plan(rows)
    pptr, pent = po.pair_union_plan(rows)
    sched, cnt = po.pair_schedule(rows)
    for got, want in ((plan.row_ptr, ptr), (plan.cols, cols), (plan.pair_ptr, pptr), (plan.pair_ent, pent),
                      (plan.sched, sched), (plan.sched_cnt, cnt)):
        assert torch.equal(got.cpu(), want)
    if not bool(better.any()):
        assert plan.pair_q is None and plan.sched_cnt_kernel is None
        return
    pq = torch.full((S, 2 * ((nbq + 1) // 2)), -1, dtype=torch.int32)
    pq[:, :nbq] = order.to(torch.int32)
    assert torch.equal(plan.pair_q.cpu().view(S, -1), pq)
    assert torch.equal(plan.sched_cnt_kernel.cpu(), cnt | ((pq.view(-1, 2) + 1) << 16))

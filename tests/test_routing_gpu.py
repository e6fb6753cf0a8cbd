"""The routing tables at the sizes where the cluster's runs, rounds and expert sweeps end unevenly: exact integers
against a stable sort, with entries that name no expert left alone."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs", [1, 31, 33, 1024, 2048, 2049, 8191, 65536 + 17, 196608])
@pytest.mark.parametrize("nexperts", [1, 8, 31, 32, 65, 1024])
def test_scatter_index_is_a_stable_sort(pairs, nexperts):
    import flux_b200 as flux

    g = torch.Generator().manual_seed(pairs + nexperts)
    chosen = (torch.rand(pairs, 1, generator=g) ** 2 * nexperts).to(torch.int32).clamp_(max=nexperts - 1)
    si, splits = flux.calc_scatter_index(chosen.cuda(), torch.empty(nexperts), return_splits=True)
    order = torch.argsort(chosen.view(-1), stable=True)
    want = torch.empty(pairs, dtype=torch.int32)
    want[order] = torch.arange(pairs, dtype=torch.int32)
    assert torch.equal(si.cpu().view(-1), want)
    assert torch.equal(splits.cpu(), torch.bincount(chosen.view(-1), minlength=nexperts).to(torch.int32))


def test_entries_without_an_expert_take_no_row():
    import flux_b200 as flux

    g = torch.Generator().manual_seed(1)
    chosen = torch.randint(-2, 12, (5000, 1), generator=g, dtype=torch.int32)
    si, splits = flux.calc_scatter_index(chosen.cuda(), torch.empty(10), return_splits=True)
    ok = (chosen.view(-1) >= 0) & (chosen.view(-1) < 10)
    rows = si.cpu().view(-1)[ok]
    order = torch.argsort(chosen.view(-1)[ok], stable=True)
    want = torch.empty_like(rows)
    want[order] = torch.arange(rows.numel(), dtype=torch.int32)
    assert torch.equal(rows, want)
    assert int(splits.sum()) == int(ok.sum())

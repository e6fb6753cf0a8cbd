"""MoE layers on one rank at sizes where the destination-order permute, the tile table and the combine end unevenly:
rows that do not fill a 32-row unit or a 256-row block, experts without rows or with all of them, more choices than
one round of the combine. Checked against the same products in 64 bits: 2^-8 of the value for the bf16 rounding of
layer 0; for layer 1 one such rounding per summed row (of that row's size) and one of the sum."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _routing(kind, tokens, experts, topk, g):
    if kind == "even":
        return torch.topk(torch.rand(tokens, experts, generator=g), topk, dim=1).indices.to(torch.int32)
    chosen = torch.arange(topk, dtype=torch.int32).repeat(tokens, 1)  # the first topk experts take everything
    if kind == "one odd":
        chosen[tokens // 2, topk - 1] = experts - 1
    return chosen


@pytest.mark.parametrize("tokens,hidden,ffn,experts,topk", [(1, 64, 8, 4, 1), (33, 1032, 72, 8, 3), (257, 2048, 264, 5, 5),
                                                            (1100, 520, 520, 64, 2), (1500, 1024, 256, 2, 1)])
@pytest.mark.parametrize("kind", ["even", "first", "one odd"])
@pytest.mark.parametrize("cta_group", [0, 2])
def test_both_layers(tokens, hidden, ffn, experts, topk, kind, cta_group):
    import flux_b200 as flux

    flux.init_flux_shm(None)
    g = torch.Generator().manual_seed(tokens + hidden)
    chosen = _routing(kind, tokens, experts, topk, g).cuda()
    gg = torch.Generator(device="cuda").manual_seed(tokens)
    x = torch.randn(tokens, hidden, generator=gg, device="cuda").to(BF16)
    ws = [(torch.randn(experts, ffn, hidden, generator=gg, device="cuda") * 0.05).to(BF16) for _ in range(2)]
    wd = (torch.randn(experts, hidden, ffn, generator=gg, device="cuda") * 0.05).to(BF16)
    vec = torch.rand(tokens * topk, generator=gg, device="cuda") + 0.5
    si, splits = flux.calc_scatter_index(chosen, torch.empty(experts), return_splits=True)
    tuning = {"cta_group": cta_group} if cta_group else None
    l0 = flux.GemmGroupedV3AGScatter(flux.DistEnvTPWithEP(None, 1, None), flux.MoeArguments(tokens, hidden, ffn, experts, topk, BF16))
    l1 = flux.GemmGroupedV3GatherRS(experts, tokens * topk, hidden, topk, 0, 1, 1, 1, input_dtype=BF16)
    gathered = torch.empty_like(x)
    outs = l0.forward_multiple_weights(x, ws, splits, si, allgather_output=gathered, tuning=tuning)
    z = l1.forward_gather_rs(outs[0], wd, splits.cpu(), si.view(-1), output_vec_scale=vec, tuning=tuning)
    torch.cuda.synchronize()
    l0.comm.check_status()
    assert torch.equal(gathered, x)
    rows = si.view(-1).long()
    token = torch.arange(tokens, device="cuda").repeat_interleave(topk)
    expert = chosen.view(-1).long()
    sums = torch.zeros(tokens, hidden, dtype=torch.float64, device="cuda")
    room = torch.zeros_like(sums)
    for e in range(experts):
        sel = expert == e
        if not bool(sel.any()):
            continue
        for out, w in zip(outs, ws):
            ref = x[token[sel]].double() @ w[e].double().t()
            slack = 2.0 ** -8 * ref.abs() + hidden * 2.0 ** -23 * (x[token[sel]].double().abs() @ w[e].double().abs().t()) + 1e-6
            assert bool(((out[rows[sel]].double() - ref).abs() <= slack).all())
        part = (outs[0][rows[sel]].double() @ wd[e].double().t()) * vec[rows[sel]][:, None].double()
        size = (outs[0][rows[sel]].double().abs() @ wd[e].double().abs().t()) * vec[rows[sel]][:, None].double()
        sums.index_add_(0, token[sel], part)
        room.index_add_(0, token[sel], 2.0 ** -8 * part.abs() + (ffn + topk) * 2.0 ** -23 * size)
    assert bool(((z.double() - sums).abs() <= room + 2.0 ** -8 * sums.abs() + 1e-6).all())


def test_calls_without_tokens_are_refused_once_none_are_kept():
    """`keep_tokens(0)` (what the Python op sets on one rank) and a call without tokens exclude one another."""
    import flux_b200 as flux
    from flux_b200 import _lib

    flux.init_flux_shm(None)
    l0 = flux.GemmGroupedV3AGScatter(flux.DistEnvTPWithEP(None, 1, None), flux.MoeArguments(8, 64, 8, 2, 1, BF16))
    x, w = torch.randn(8, 64, device="cuda").to(BF16), torch.randn(2, 8, 64, device="cuda").to(BF16)
    si, splits = flux.calc_scatter_index(torch.zeros(8, 1, dtype=torch.int32, device="cuda"), torch.empty(2), return_splits=True)
    out = l0.forward(x, w, splits, si)
    args = (8, w.data_ptr(), splits.data_ptr(), si.data_ptr(), None, out.data_ptr(), None, None, torch.cuda.current_stream().cuda_stream)
    lib = _lib.load()
    with pytest.raises(_lib.FluxbError):
        _lib.check(lib.fluxb_moe_ag_scatter_forward(l0._h, None, *args))
    _lib.check(lib.fluxb_moe_ag_scatter_keep_tokens(l0._h, 1))
    want = l0.forward(x, w, splits, si).clone()
    out.zero_()
    _lib.check(lib.fluxb_moe_ag_scatter_forward(l0._h, None, *args))
    torch.cuda.synchronize()
    assert torch.equal(out, want)

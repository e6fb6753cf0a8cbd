"""Launches that may become resident while the launch before them still runs (programmatic dependent launch)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


@pytest.fixture()
def flux():
    import flux_b200

    flux_b200.init_flux_shm(None)
    yield flux_b200
    flux_b200.get_comm(None).set_timeout_ms(5000)


@pytest.mark.parametrize("m,bias", [(16, "none"), (512, "none"), (512, "unaligned")])  # few rows, plain, fused kernel
def test_the_wait_budget_starts_when_the_launch_before_has_ended(flux, m, bias):
    """One CTA works through 2048 tiles (about 70 ms) and leaves 147 SMs free for the next launch, whose waits may last
    10 ms: they are not to be counted from the moment it became resident."""
    n = k = 512
    g = torch.Generator(device="cuda").manual_seed(m)
    big = torch.zeros(8192, 8192, device="cuda", dtype=BF16)
    sink = torch.empty_like(big)
    a = torch.randn(m, k, generator=g, device="cuda").to(BF16)
    b = (torch.randn(n, k, generator=g, device="cuda") * 0.02).to(BF16)
    t = None if bias == "none" else torch.randn(n + 1, generator=g, device="cuda").to(BF16)[1:].view(1, n)
    op = flux.GemmOnly(BF16)
    long_tuning = {"block_n": 256, "cta_group": 1, "num_ctas": 1}
    op.forward(big[:256], big[:256], tuning=long_tuning)
    want = op.forward(a, b, bias=t)
    torch.cuda.synchronize()
    flux.get_comm(None).set_timeout_ms(10)
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    start.record()
    op.forward(big, big, output_buf=sink, tuning=long_tuning)
    out = op.forward(a, b, bias=t)
    end.record()
    torch.cuda.synchronize()
    flux.get_comm(None).check_status()
    assert start.elapsed_time(end) > 30, "the first launch is meant to last several budgets"
    assert torch.equal(out, want)

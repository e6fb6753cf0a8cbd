"""Launches that may become resident while the launch before them still runs (programmatic dependent launch)."""
import ctypes as C
import os
import sys

import pytest
import torch

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from ranks_on_gpu import Ranks, _p, _stream  # noqa: E402

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


def test_nothing_starts_beside_a_launch_that_waits_for_a_peer(flux):
    """Rank 0 of two runs alone and gives up on its peer after 300 ms; most of its CTAs have nothing to do by then.
    A plain GEMM behind it enters the GPU only when it has ended (and is not disturbed by it)."""
    from flux_b200 import _lib

    lib, n, k, m_local = _lib.load(), 256, 512, 128
    g = torch.Generator(device="cuda").manual_seed(7)
    a = torch.randn(512, k, generator=g, device="cuda").to(BF16)
    b = (torch.randn(n, k, generator=g, device="cuda") * 0.02).to(BF16)
    op = flux.GemmOnly(BF16)
    want = op.forward(a, b)
    comm = flux.get_comm(None)
    comm.set_timeout_ms(100)
    words = torch.cuda.get_device_properties(0).multi_processor_count * 8
    first, second = (torch.zeros(words, dtype=torch.int64, device="cuda") for _ in range(2))
    rk = Ranks(2, timeout_ms=300)
    try:
        ops = rk.ag_gemm_ops(2 * m_local, n, k, BF16, BF16)
        gathered = torch.zeros(2 * m_local, n, dtype=BF16, device="cuda")
        _lib.check(lib.fluxb_comm_set_ranks_on_gpu(rk.comms[0], 1))
        _lib.check(lib.fluxb_comm_set_trace(rk.comms[0], _p(first)))
        _lib.check(lib.fluxb_comm_set_trace(comm.handle, _p(second)))
        _lib.check(lib.fluxb_ag_gemm_forward(ops[0], _p(a), m_local, _p(b), n, k, _p(gathered), None, 0, None, None, 1.0, 0, None,
                                             None, _stream()))
        out = op.forward(a, b)
        torch.cuda.synchronize()
        status = C.c_int(-1)
        _lib.check(lib.fluxb_status_peek(rk.comms[0], C.byref(status)))
        assert status.value == 5  # the wait for the peer's rows ran out
        comm.check_status()
        assert torch.equal(out, want)
        entered = second.view(-1, 8)[:, 0]
        assert int(entered[entered > 0].min()) >= int(first.view(-1, 8)[:, 3:5].max())
    finally:
        _lib.check(lib.fluxb_comm_set_trace(comm.handle, None))
        rk.close()


@pytest.mark.parametrize("m", [16, 512])  # few rows, plain
def test_with_several_ranks_no_gemm_starts_early(flux, m):
    """Behind a launch that lets the next one in early (one CTA, several ms), a GEMM of a rank of two waits outside."""
    from flux_b200 import _lib

    lib, n, k = _lib.load(), 256, 512
    a, b = torch.ones(m, k, device="cuda", dtype=BF16), torch.ones(n, k, device="cuda", dtype=BF16)
    out = torch.empty(m, n, device="cuda", dtype=BF16)
    big = torch.zeros(2048, 8192, device="cuda", dtype=BF16)
    comm = flux.get_comm(None)
    words = torch.cuda.get_device_properties(0).multi_processor_count * 8
    first, second = (torch.zeros(words, dtype=torch.int64, device="cuda") for _ in range(2))
    two = C.c_void_p()
    _lib.check(lib.fluxb_comm_create(0, 2, C.byref(two)))
    try:
        _lib.check(lib.fluxb_comm_set_trace(comm.handle, _p(first)))
        _lib.check(lib.fluxb_comm_set_trace(two, _p(second)))
        for _ in range(2):  # the first round loads the kernels
            flux.GemmOnly(BF16).forward(big, big, tuning={"block_n": 256, "cta_group": 1, "num_ctas": 1})
            _lib.check(lib.fluxb_gemm(two, _p(a), _p(b), _p(out), m, n, k, _lib.BF16, _lib.BF16, None, 0, None, None, 1.0, 0, None,
                                      _stream()))
            torch.cuda.synchronize()
        assert bool((out == k).all())
        entered = second.view(-1, 8)[:, 0]
        assert int(entered[entered > 0].min()) >= int(first.view(-1, 8)[0, 3])
    finally:
        _lib.check(lib.fluxb_comm_set_trace(comm.handle, None))
        lib.fluxb_comm_destroy(two)

"""The plain GEMM's epilogue and split last wave at the sizes and options where they can go wrong: rows and columns
that end inside a warp's 32 rows or a 64-column box, vectors that are not 16-byte aligned, K cut over several CTAs.

Bound of every element: half a unit in the last place of the 16-bit output, taken twice (2^-8 of the value for bf16,
2^-11 for fp16), plus K roundings of fp32 sums, K * 2^-23 * sum |a| |b|. int8 is compared bit for bit."""
import ctypes as C
import time

import pytest
import torch

pytestmark = pytest.mark.gpu
BF16, FP16 = torch.bfloat16, torch.float16


@pytest.fixture(scope="module")
def flux():
    import flux_b200

    flux_b200.init_flux_shm(None)
    flux_b200.get_comm(None).set_timeout_ms(5000)
    return flux_b200


def _inputs(m, n, k, dtype, seed=5):
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randn(m, k, generator=g, device="cuda").to(dtype)
    b = (torch.randn(n, k, generator=g, device="cuda") * 0.02).to(dtype)
    return a, b, g


def _check(flux, out, a, b, extra=None):
    torch.cuda.synchronize()
    flux.get_comm(None).check_status()
    ref = a.double() @ b.double().t()
    if extra is not None:
        ref = ref + extra.double()
    bound = ref.abs() * (2.0 ** -8 if out.dtype == BF16 else 2.0 ** -11)
    bound += a.shape[1] * 2.0 ** -23 * (a.double().abs() @ b.double().abs().t()) + 1e-6
    worst = ((out.double() - ref).abs() / bound).max().item()
    assert worst <= 1.0, f"{worst:.2f} times the bound"


@pytest.mark.parametrize("dtype", [BF16, FP16])
@pytest.mark.parametrize("m,n,k,tuning", [
    (1, 8, 64, None), (31, 72, 128, None), (33, 56, 512, None), (289, 328, 320, {"cta_group": 2}), (300, 200, 192, {"cta_group": 1}),
    (130, 264, 512, {"block_n": 64, "cta_group": 1}), (257, 512, 1024, {"block_n": 256, "cta_group": 2}),
])
@pytest.mark.parametrize("bias", ["none", "row", "full", "row unaligned", "full unaligned"])
def test_epilogue_edges(flux, m, n, k, tuning, bias, dtype):
    a, b, g = _inputs(m, n, k, dtype)
    rows = m if bias.startswith("full") else 1
    t = None
    if bias != "none":
        flat = torch.randn(rows * n + 1, generator=g, device="cuda").to(dtype)
        t = (flat[1:] if "unaligned" in bias else flat[:-1]).view(rows, n)
    out = flux.GemmOnly(dtype).forward(a, b, bias=t, tuning=tuning)
    _check(flux, out, a, b, t)


# (rows, columns, bytes of K) that get 256 x 512 tiles: 16 x 14 of them, three waves of 74 pairs and a cut rest
WIDE_SHAPES = [(4000, 7160, 16384), (4096, 7168, 16384)]


@pytest.fixture()
def wide(flux):
    """Asserts that the test's last launch had at most four work items a CTA: 256 x 256 tiles would have had seven."""
    lib, comm = flux._lib.load(), flux.get_comm(None)
    stamps = torch.zeros(torch.cuda.get_device_properties(0).multi_processor_count, 8, dtype=torch.int64, device="cuda")
    flux._lib.check(lib.fluxb_comm_set_trace(comm.handle, stamps.data_ptr()))
    yield
    flux._lib.check(lib.fluxb_comm_set_trace(comm.handle, None))
    torch.cuda.synchronize()
    assert 3 <= int(stamps[:, 7].max()) <= 4


@pytest.mark.parametrize("kn", [False, True])
@pytest.mark.parametrize("shape,bias", list(zip(WIDE_SHAPES, ("row", "full"))))
def test_wide_tiles(flux, wide, shape, bias, kn):
    """Rows and columns that end inside a tile, and whole ones."""
    m, n, _ = shape
    a, b, g = _inputs(m, n, 8192, BF16)
    t = torch.randn(1 if bias == "row" else m, n, generator=g, device="cuda").to(BF16)
    out = flux.GemmOnly(BF16, transpose_weight=kn).forward(a, b.t().contiguous() if kn else b, bias=t)
    _check(flux, out, a, b, t)


@pytest.mark.parametrize("shape", WIDE_SHAPES)
def test_wide_tiles_fp8(flux, wide, shape):
    m, n, k = shape
    g = torch.Generator(device="cuda").manual_seed(10)
    a, b = (torch.randn(r, k, generator=g, device="cuda").to(torch.float8_e4m3fn) for r in (m, n))
    sa, sb = (torch.rand(r, generator=g, device="cuda") * 0.01 + 0.001 for r in (m, n))
    out = flux.GemmOnly(torch.float8_e4m3fn).forward(a, b, input_scale=sa, weight_scale=sb)
    _check(flux, out, a.double() * sa[:, None].double(), b.double() * sb[:, None].double())


@pytest.mark.parametrize("shape", WIDE_SHAPES)
def test_wide_tiles_int8(flux, wide, shape):
    m, n, k = shape
    g = torch.Generator(device="cuda").manual_seed(9)
    a = torch.randint(-127, 128, (m, k), generator=g, device="cuda", dtype=torch.int32).to(torch.int8)
    b = torch.randint(-127, 128, (n, k), generator=g, device="cuda", dtype=torch.int32).to(torch.int8)
    one_m, one_n = torch.ones(m, device="cuda"), torch.ones(n, device="cuda")
    out = flux.GemmOnly(torch.int8).forward(a, b, input_scale=one_m, weight_scale=one_n)
    torch.cuda.synchronize()
    assert torch.equal(out, (a.double() @ b.double().t()).float().to(BF16))


def test_tile_widths_a_caller_may_not_choose(flux):
    a, b, _ = _inputs(512, 512, 256, BF16)
    for width in (96, 512):
        with pytest.raises(Exception):
            flux.GemmOnly(BF16).forward(a, b, tuning={"block_n": width})


@pytest.mark.parametrize("kn", [False, True])
@pytest.mark.parametrize("m", [1, 2, 16, 17, 32, 33, 64, 65, 128, 129, 256])
@pytest.mark.parametrize("n,k", [(8, 64), (136, 264), (1160, 4096), (5000, 1032)])  # cut along K into 1, 1, 8 or 4, 4 or 2 parts
def test_few_rows(flux, m, n, k, kn):
    a, b, g = _inputs(m, n, k, BF16, seed=m + n)
    bias = torch.randn(m if m % 2 else 1, n, generator=g, device="cuda").to(BF16)
    out = flux.GemmOnly(BF16, transpose_weight=kn).forward(a, b.t().contiguous() if kn else b, bias=bias)
    _check(flux, out, a, b, bias)


@pytest.mark.parametrize("m", [3, 40, 100, 200])
def test_few_rows_8bit(flux, m):
    n, k = 1288, 4112
    g = torch.Generator(device="cuda").manual_seed(m)
    sa, sb = torch.rand(m, generator=g, device="cuda") * 0.01 + 0.001, torch.rand(n, generator=g, device="cuda") * 0.01 + 0.001
    ai = torch.randint(-127, 128, (m, k), generator=g, device="cuda", dtype=torch.int32).to(torch.int8)
    bi = torch.randint(-127, 128, (n, k), generator=g, device="cuda", dtype=torch.int32).to(torch.int8)
    bias = torch.randn(1, n, generator=g, device="cuda").to(BF16)
    out = flux.GemmOnly(torch.int8).forward(ai, bi, bias=bias, input_scale=sa, weight_scale=sb)
    torch.cuda.synchronize()
    acc = (ai.double() @ bi.double().t()).float()
    assert torch.equal(out, ((sa[:, None] * sb[None, :]) * acc).to(BF16) + bias)
    a8, b8 = torch.randn(m, k, generator=g, device="cuda").to(torch.float8_e4m3fn), torch.randn(n, k, generator=g, device="cuda").to(torch.float8_e4m3fn)
    out = flux.GemmOnly(torch.float8_e4m3fn).forward(a8, b8, input_scale=sa, weight_scale=sb)
    _check(flux, out, a8.double() * sa[:, None].double(), b8.double() * sb[:, None].double())


def test_few_rows_on_two_streams(flux):
    """Launches that run side by side share nothing: same result as one after the other."""
    a, b, _ = _inputs(16, 2048, 4096, BF16)
    a2 = a.flip(0).contiguous()
    op = flux.GemmOnly(BF16)
    want, want2 = op.forward(a, b), op.forward(a2, b)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    outs = [[], []]
    for _ in range(20):
        for i, x in enumerate((a, a2)):
            with torch.cuda.stream(streams[i]):
                outs[i].append(op.forward(x, b))
    torch.cuda.synchronize()
    assert all(torch.equal(o, want) for o in outs[0]) and all(torch.equal(o, want2) for o in outs[1])


@pytest.mark.parametrize("shift", [0, 1])
def test_column_scales_of_any_alignment(flux, shift):
    m, n, k = 200, 264, 256
    g = torch.Generator(device="cuda").manual_seed(3)
    a = torch.randint(-127, 128, (m, k), generator=g, device="cuda", dtype=torch.int32).to(torch.int8)
    b = torch.randint(-127, 128, (n, k), generator=g, device="cuda", dtype=torch.int32).to(torch.int8)
    sa = torch.rand(m, generator=g, device="cuda") * 0.01 + 0.001
    sb = (torch.rand(n + 1, generator=g, device="cuda") * 0.01 + 0.001)[shift:n + shift]
    out = flux.GemmOnly(torch.int8).forward(a, b, input_scale=sa, weight_scale=sb)
    torch.cuda.synchronize()
    acc = (a.double() @ b.double().t()).float()  # exact: below 2^24
    assert torch.equal(out, ((sa[:, None] * sb[None, :]) * acc).to(BF16))


@pytest.mark.parametrize("m,n,tuning", [(130, 72 + 64 * 4, {"block_n": 64, "cta_group": 1, "num_ctas": 8}),
                                        (300, 1288, {"block_n": 256, "cta_group": 2, "num_ctas": 16})])
def test_int8_accumulators_cut_along_k_stay_whole_numbers(flux, m, n, tuning):
    k = 8192  # 64 K blocks; 12 tiles on 8 workers: the last 4 (two) are cut into 2 (four) parts
    g = torch.Generator(device="cuda").manual_seed(4)
    a = torch.randint(-127, 128, (m, k), generator=g, device="cuda", dtype=torch.int32).to(torch.int8)
    b = torch.randint(-127, 128, (n, k), generator=g, device="cuda", dtype=torch.int32).to(torch.int8)
    ones_m, ones_n = torch.ones(m, device="cuda"), torch.ones(n, device="cuda")
    for _ in range(2):  # the counters of the parts clear themselves
        out = flux.GemmOnly(torch.int8).forward(a, b, input_scale=ones_m, weight_scale=ones_n, tuning=tuning)
        torch.cuda.synchronize()
        flux.get_comm(None).check_status()
        assert torch.equal(out, (a.double() @ b.double().t()).float().to(BF16))


class _OwnComm:
    """A communicator without any stream's scratch taken yet."""

    def __init__(self):
        from flux_b200 import _lib

        self.lib, self.handle = _lib.load(), C.c_void_p()
        _lib.check(self.lib.fluxb_comm_create(0, 1, C.byref(self.handle)))
        _lib.check(self.lib.fluxb_comm_set_timeout_ms(self.handle, 5000))

    def check_status(self):
        torch.cuda.synchronize()
        status = C.c_int(-1)
        assert self.lib.fluxb_status_peek(self.handle, C.byref(status)) == 0 and status.value == 0

    def __del__(self):
        self.lib.fluxb_comm_destroy(self.handle)


def _cut_launch(flux, dtype, num_ctas):
    """38 tiles of 256 x 256: one is left to be cut into 8 parts on 37 CTA pairs (74 CTAs), two on 18 (36 CTAs)."""
    g = torch.Generator(device="cuda").manual_seed(11)
    m, n, k, tuning = 512, 19 * 256, 16384, {"block_n": 256, "cta_group": 2, "num_ctas": num_ctas}
    if dtype == torch.int8:
        a, a2, b = (torch.randint(-127, 128, (r, k), generator=g, device="cuda", dtype=torch.int32).to(torch.int8) for r in (m, m, n))
        kw = {"input_scale": torch.ones(m, device="cuda"), "weight_scale": torch.ones(n, device="cuda")}
    else:
        a, a2, b = (torch.randn(r, k, generator=g, device="cuda").to(dtype) for r in (m, m, n))
        kw = {}
    op = flux.GemmOnly(dtype)
    op.comm = _OwnComm()
    return op.comm, a, a2, lambda x, out=None, bias=None: op.forward(x, b, output_buf=out, bias=bias, tuning=tuning, **kw)


@pytest.mark.parametrize("kernel", ["plain", "fused"])
@pytest.mark.parametrize("dtype", [BF16, torch.int8])
def test_cut_launches_on_two_streams(flux, dtype, kernel):
    """Two launches side by side on half the SMs each, each with parts of its own last wave: the results of one after the
    other. (An unaligned bias takes the fused kernel.)"""
    comm, a, a2, call = _cut_launch(flux, dtype, 74)
    bias = None if kernel == "plain" else torch.ones(19 * 256 + 1, device="cuda", dtype=BF16)[1:].view(1, -1)
    want = [call(a, bias=bias), call(a2, bias=bias)]
    comm.check_status()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    outs = [[], []]
    for _ in range(20):
        for i, x in enumerate((a, a2)):
            with torch.cuda.stream(streams[i]):
                outs[i].append(call(x, bias=bias))
    comm.check_status()
    for i in range(2):
        assert all(torch.equal(o, want[i]) for o in outs[i])


def test_cut_launches_in_graphs_beside_eager_ones(flux):
    """Two graphs captured on one stream, replayed on two others beside eager launches on that stream."""
    comm, a, a2, call = _cut_launch(flux, BF16, 36)
    want, want2 = call(a), call(a2)
    outs = [torch.empty_like(want) for _ in range(3)]
    side = [torch.cuda.Stream() for _ in range(3)]
    comm.check_status()
    graphs = [torch.cuda.CUDAGraph() for _ in range(2)]
    for graph, x, out in zip(graphs, (a, a2), outs):
        with torch.cuda.graph(graph, stream=side[2]):
            call(x, out)
    for _ in range(10):
        for i in range(2):
            with torch.cuda.stream(side[i]):
                graphs[i].replay()
        with torch.cuda.stream(side[2]):
            call(a, outs[2])
    comm.check_status()
    assert torch.equal(outs[0], want) and torch.equal(outs[1], want2) and torch.equal(outs[2], want)


def test_eager_cut_launch_while_another_stream_captures(flux):
    """The stream that a launch goes to is asked for its identity without disturbing a capture on another one."""
    comm, a, a2, call = _cut_launch(flux, BF16, 74)
    want, want2 = call(a), call(a2)
    outs = [torch.empty_like(want) for _ in range(2)]
    eager, stream, graph = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    comm.check_status()
    with torch.cuda.graph(graph, stream=stream):
        call(a, outs[0])
        with torch.cuda.stream(eager):
            call(a2, outs[1])
    graph.replay()
    comm.check_status()
    assert torch.equal(outs[0], want) and torch.equal(outs[1], want2)


def test_graphs_give_their_scratch_back(flux):
    """More graphs, one after the other, than there is scratch for: the last is cut like the first (the same sums)."""
    comm, a, _, call = _cut_launch(flux, BF16, 74)
    want = call(a)
    stream = torch.cuda.Stream()
    for _ in range(12):
        out = torch.empty_like(want)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            call(a, out)
        graph.replay()
        comm.check_status()
        assert torch.equal(out, want)
        del graph
        time.sleep(0.1)  # the driver gives it back from a thread of its own


def test_more_streams_than_scratch(flux):
    """Streams that come when all scratch is taken run uncut; whole-number sums are the same."""
    comm, a, _, call = _cut_launch(flux, torch.int8, 74)
    want = call(a)
    outs = []
    for stream in [torch.cuda.Stream() for _ in range(20)]:
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            outs.append(call(a))
    comm.check_status()
    assert all(torch.equal(o, want) for o in outs)


def test_timeline_has_room_for_one_cta_per_sm(flux):
    """Few rows run up to two CTAs on an SM; the timeline buffer holds one per SM, and nothing is written behind it."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    m, n, k = 16, 128 * sms, 1024  # one tile per SM, cut in two: twice as many CTAs as SMs
    a, b, _ = _inputs(m, n, k, BF16)
    lib, comm = flux._lib.load(), flux.get_comm(None)
    stamps = torch.zeros(4 * sms, 8, dtype=torch.int64, device="cuda")
    flux._lib.check(lib.fluxb_comm_set_trace(comm.handle, stamps.data_ptr()))
    try:
        out = flux.GemmOnly(BF16).forward(a, b)
    finally:
        flux._lib.check(lib.fluxb_comm_set_trace(comm.handle, None))
    _check(flux, out, a, b)
    assert bool((stamps[:sms, 0] > 0).all()) and not bool(stamps[sms:].any())


def test_misaligned_vectors_are_refused(flux):
    """The kernels move output rows and MoE tokens 16 bytes at a time: anything else is an error of the call, unless the few-row
    kernel (4 bytes) takes it."""
    m, n, k = 300, 64, 128
    a, b, g = _inputs(m, n, k, BF16)
    shifted = lambda rows, cols, by: torch.zeros(rows * cols + by, dtype=BF16, device="cuda")[by:].view(rows, cols)
    op = flux.GemmOnly(BF16)
    for by in (1, 2, 4):
        with pytest.raises(RuntimeError, match="aligned"):
            op.forward(a, b, output_buf=shifted(m, n, by))
    with pytest.raises(RuntimeError, match="aligned"):
        op.forward(a[:16], b, output_buf=shifted(16, n, 1))
    out = op.forward(a[:16], b, output_buf=shifted(16, n, 2))
    _check(flux, out, a[:16], b)
    tokens, experts, topk = 8, 2, 2
    si, splits = flux.calc_scatter_index(torch.tensor([[0, 1]] * tokens, dtype=torch.int32, device="cuda"), torch.empty(2), return_splits=True)
    l0 = flux.GemmGroupedV3AGScatter(flux.DistEnvTPWithEP(None, 1, None), flux.MoeArguments(tokens, k, n, experts, topk, BF16))
    w = torch.zeros(experts, n, k, dtype=BF16, device="cuda")
    with pytest.raises(RuntimeError, match="tokens must be 16-byte aligned"):
        l0.forward(shifted(tokens, k, 1), w, splits, si)
    with pytest.raises(RuntimeError, match="output must be 16-byte aligned"):
        l0.forward(a[:tokens], w, splits, si, outputs_buf=shifted(tokens * topk, n, 1))

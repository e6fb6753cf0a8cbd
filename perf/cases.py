"""The workloads this framework is timed on, as one GPU sees them.

Every case is a call, or a short chain of calls, that a tensor-parallel layer makes through the public entry
points of `flux_b200`, at the sizes of one rank's share of the layer (N / TP or K / TP columns; the shares of the
configurations that `bench.py` and the tests name, and sizes between them):

  gemm    `GemmOnly.forward`: the unfused building block, all data types and options
  mlp     `AGKernel.forward` followed by `GemmRS.forward` on its result: the dense MLP of one layer, from a single
          decoded token to a full prefill batch
  ag      `AGKernel.forward` alone with quantised inputs (fp8 per-row x per-channel scales)
  train   `layers.TensorParallelMLP`, forward and backward: the gradients of the input and of all parameters
  moe     `GemmGroupedV3AGScatter.forward` and `GemmGroupedV3GatherRS.forward_gather_rs` over a given routing
  layer   `layers.MoEMLP.forward`: router, routing tables, both grouped layers
  route   `calc_scatter_index` and `calc_gather_index`: the routing tables of one batch

`prepare` makes what a program holds before the call (weights, activations, op objects with their buffers); `run`
is one pass. Activations are N(0, 1), weights N(0, 0.02), routing logits N(0, 1), as in the tests and the
benchmark.
"""
import math

import torch

import flux_b200 as flux
from flux_b200 import layers

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp8": torch.float8_e4m3fn, "int8": torch.int8}


def listed():
    return [
        # the reference test's smallest shape: the call itself costs more than its arithmetic
        {"name": "gemm_smallest", "kind": "gemm", "dtype": "bf16", "m": 256, "n": 512, "k": 512, "bias": "none", "weight_kn": False},
        # routing tables of one prefill batch, 8 experts top-2
        {"name": "route_prefill", "kind": "route", "tokens": 8192, "experts": 8, "topk": 2},
        # decoding one sequence: every weight is read for one token (an eighth of hidden 8192, ffn 28672)
        {"name": "mlp_decode_one", "kind": "mlp", "dtype": "fp16", "m": 1, "hidden": 8192, "ffn": 3584, "bias": "none"},
        # decoding a batch (an eighth of hidden 12288, ffn 49152)
        {"name": "mlp_decode_batch", "kind": "mlp", "dtype": "bf16", "m": 48, "hidden": 12288, "ffn": 6144, "bias": "none"},
        # a ragged chunk of a prompt, with biases (a quarter of hidden 4096, ffn 14336)
        {"name": "mlp_chunk_ragged", "kind": "mlp", "dtype": "bf16", "m": 1000, "hidden": 4096, "ffn": 3584, "bias": "row"},
        # the benchmark's dense layer, undivided
        {"name": "mlp_prefill_full", "kind": "mlp", "dtype": "bf16", "m": 4096, "hidden": 12288, "ffn": 49152, "bias": "none"},
        # the fp8 configuration (a quarter of N=28672)
        {"name": "fp8_prefill", "kind": "ag", "dtype": "fp8", "m": 8192, "n": 7168, "k": 8192},
        # w8a8 inference of a ragged batch: per-row x per-channel dequantisation and a bias
        {"name": "w8a8_ragged", "kind": "gemm", "dtype": "int8", "m": 2000, "n": 6144, "k": 12288, "bias": "row", "weight_kn": False},
        # a training step of a dense MLP block with biases
        {"name": "mlp_train_step", "kind": "train", "dtype": "bf16", "m": 2048, "hidden": 4096, "ffn": 14336, "bias": True},
        # the MoE configuration (a quarter of ffn 14336): 8192 tokens, 8 experts, top-2
        {"name": "moe_prefill", "kind": "moe", "dtype": "bf16", "tokens": 8192, "hidden": 4096, "ffn": 3584, "experts": 8, "topk": 2},
        # many small experts, ragged, quantised: 32 experts top-4 (an eighth of ffn 8192)
        {"name": "moe_fine_fp8", "kind": "moe", "dtype": "fp8", "tokens": 2000, "hidden": 8192, "ffn": 1024, "experts": 32, "topk": 4},
        # decoding a batch through a whole gated MoE layer (a quarter of ffn 14336)
        {"name": "moe_layer_decode", "kind": "layer", "dtype": "bf16", "tokens": 64, "hidden": 4096, "ffn": 3584, "experts": 8, "topk": 2, "gated": True},
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of `step` between lo and hi, spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(max(int(round(v / step)) * step, lo), hi))


def draw(rng):
    kind = rng.choice(["gemm", "gemm", "mlp", "mlp", "mlp", "ag", "train", "moe", "moe", "layer", "route"])
    if kind == "gemm":
        dtype = rng.choice(["bf16", "fp16", "fp8", "int8"])
        step = 8 if dtype in ("bf16", "fp16") else 16
        return {"kind": kind, "dtype": dtype, "m": _log(rng, 1, 8192), "n": _log(rng, 512, 12288, 8), "k": _log(rng, 512, 12288, step),
                "bias": rng.choice(["none", "row"] + (["full"] if dtype in ("bf16", "fp16") else [])),
                "weight_kn": dtype in ("bf16", "fp16") and rng.random() < 0.3}
    if kind == "mlp":
        return {"kind": kind, "dtype": rng.choice(["bf16", "bf16", "fp16"]), "m": _log(rng, 1, 4096), "hidden": rng.choice([4096, 5120, 8192, 12288]),
                "ffn": _log(rng, 1024, 16384, 8), "bias": rng.choice(["none", "none", "row"])}
    if kind == "ag":
        return {"kind": kind, "dtype": "fp8", "m": _log(rng, 16, 8192), "n": _log(rng, 1024, 14336, 8), "k": _log(rng, 2048, 12288, 16)}
    if kind == "train":
        return {"kind": kind, "dtype": "bf16", "m": _log(rng, 256, 4096), "hidden": rng.choice([2048, 4096, 5120]), "ffn": _log(rng, 1024, 14336, 8),
                "bias": rng.random() < 0.5}
    experts = rng.choice([8, 16, 32, 64])
    topk = rng.choice([1, 2, 4]) if experts < 32 else rng.choice([2, 4, 6])
    if kind == "moe":
        return {"kind": kind, "dtype": rng.choice(["bf16", "bf16", "fp8"]), "tokens": _log(rng, 32, 8192), "hidden": rng.choice([2048, 4096, 8192]),
                "ffn": _log(rng, 512, 3584, 16), "experts": experts, "topk": topk}
    if kind == "layer":
        return {"kind": kind, "dtype": "bf16", "tokens": _log(rng, 1, 4096), "hidden": rng.choice([2048, 4096]), "ffn": _log(rng, 512, 3584, 8),
                "experts": experts, "topk": topk, "gated": rng.random() < 0.5}
    return {"kind": kind, "tokens": _log(rng, 64, 32768), "experts": experts, "topk": topk}


class _Maker:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed))

    def normal(self, *shape, std=1.0, dtype=torch.bfloat16):
        t = torch.randn(shape, generator=self.g, device="cuda", dtype=torch.float32 if dtype == torch.float32 else dtype)
        return t if std == 1.0 else t.mul_(std)

    def fp8_rows(self, rows, cols, std=1.0):
        """Values quantised row by row to e4m3 and their scales, a block of rows at a time."""
        q = torch.empty((rows, cols), dtype=torch.float8_e4m3fn, device="cuda")
        s = torch.empty((rows,), dtype=torch.float32, device="cuda")
        for r in range(0, rows, 4096):
            x = torch.randn((min(4096, rows - r), cols), generator=self.g, device="cuda") * std
            sc = x.abs().amax(dim=1).clamp_min(1e-12) / 448.0
            s[r:r + 4096] = sc
            q[r:r + 4096] = (x / sc[:, None]).to(torch.float8_e4m3fn)
        return q, s

    def int8_rows(self, rows, cols, std=1.0):
        x = torch.randn((rows, cols), generator=self.g, device="cuda") * std
        s = x.abs().amax(dim=1).clamp_min(1e-12) / 127.0
        return (x / s[:, None]).round().clamp(-127, 127).to(torch.int8), s

    def routing(self, tokens, experts, topk):
        logits = torch.randn((tokens, experts), generator=self.g, device="cuda")
        w, chosen = torch.topk(torch.softmax(logits, -1), topk, dim=-1)
        return chosen.to(torch.int32), w


def prepare(case, seed):
    flux.init_flux_shm(None)
    mk = _Maker(seed)
    kind = case["kind"]
    st = {"case": case}
    dt = DTYPES.get(case.get("dtype"))
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        out = torch.bfloat16 if dt in (torch.int8, torch.float8_e4m3fn) else dt
        if dt == torch.int8:
            st["a"], st["sa"] = mk.int8_rows(m, k)
            st["b"], st["sb"] = mk.int8_rows(n, k, 0.02)
        elif dt == torch.float8_e4m3fn:
            st["a"], st["sa"] = mk.fp8_rows(m, k)
            st["b"], st["sb"] = mk.fp8_rows(n, k, 0.02)
        else:
            st["a"], st["sa"], st["sb"] = mk.normal(m, k, dtype=dt), None, None
            st["b"] = mk.normal(*((k, n) if case["weight_kn"] else (n, k)), std=0.02, dtype=dt)
        st["bias"] = None if case["bias"] == "none" else mk.normal(*((1, n) if case["bias"] == "row" else (m, n)), std=0.1, dtype=out)
        st["op"] = flux.GemmOnly(dt, transpose_weight=bool(case["weight_kn"]))
    elif kind == "mlp":
        m, h, f = case["m"], case["hidden"], case["ffn"]
        st["x"] = mk.normal(m, h, dtype=dt)
        st["w0"], st["w1"] = mk.normal(f, h, std=0.02, dtype=dt), mk.normal(h, f, std=0.02, dtype=dt)
        row = case["bias"] == "row"
        st["b0"], st["b1"] = (mk.normal(1, f, std=0.1, dtype=dt), mk.normal(1, h, std=0.1, dtype=dt)) if row else (None, None)
        st["ag"] = flux.AGKernel(None, 1, m, f, h, dt)
        st["rs"] = flux.GemmRS(None, 1, m, h, dt)
    elif kind == "ag":
        m, n, k = case["m"], case["n"], case["k"]
        st["a"], st["sa"] = mk.fp8_rows(m, k)
        st["b"], st["sb"] = mk.fp8_rows(n, k, 0.02)
        st["op"] = flux.AGKernel(None, 1, m, n, k, dt)
    elif kind == "train":
        st["mlp"] = layers.TensorParallelMLP(case["hidden"], case["ffn"], case["m"], None, case["bias"], dtype=dt)
        with torch.no_grad():
            for p in st["mlp"].parameters():
                p.copy_(mk.normal(*p.shape, std=0.02, dtype=dt))
        st["x"] = mk.normal(case["m"], case["hidden"], dtype=dt).requires_grad_(True)
        st["dy"] = mk.normal(case["m"], case["hidden"], dtype=dt)
        st["params"] = [st["x"]] + list(st["mlp"].parameters())
    elif kind == "moe":
        t, h, f, e, k = (case[x] for x in ("tokens", "hidden", "ffn", "experts", "topk"))
        chosen, w = mk.routing(t, e, k)
        st["si"], st["splits"] = flux.calc_scatter_index(chosen, torch.empty(e, dtype=torch.int32), return_splits=True)
        gi, ti = flux.calc_gather_index(st["si"])
        st["vec"] = w.reshape(-1)[gi.long() * k + ti.long()].float().contiguous()
        st["splits_cpu"] = st["splits"].cpu()
        if dt == torch.float8_e4m3fn:
            # tensor-wise scales per expert; the activations between the layers arrive quantised too
            st["x"], st["act"] = mk.normal(t, h).to(dt), mk.normal(t * k, f).to(dt)
            st["w0"] = torch.empty((e, f, h), dtype=dt, device="cuda")
            st["w1"] = torch.empty((e, h, f), dtype=dt, device="cuda")
            for i in range(e):
                st["w0"][i] = mk.normal(f, h, std=64.0).to(dt)
                st["w1"][i] = mk.normal(h, f, std=64.0).to(dt)
            st["scale0"] = torch.rand((e,), generator=mk.g, device="cuda") * 2e-4 + 2e-4
            st["scale1"] = torch.rand((e,), generator=mk.g, device="cuda") * 2e-4 + 2e-4
            st["in_scale"] = torch.full((1,), 0.5, device="cuda")
        else:
            st["x"], st["act"] = mk.normal(t, h, dtype=dt), None
            st["w0"], st["w1"] = mk.normal(e, f, h, std=0.02, dtype=dt), mk.normal(e, h, f, std=0.02, dtype=dt)
            st["scale0"] = st["scale1"] = st["in_scale"] = None
        env = flux.DistEnvTPWithEP(None, 1, None)
        st["l0"] = flux.GemmGroupedV3AGScatter(env, flux.MoeArguments(t, h, f, e, k, dt, torch.bfloat16))
        st["l1"] = flux.GemmGroupedV3GatherRS(e, t * k, h, k, 0, 1, 1, 1, input_dtype=dt)
    elif kind == "layer":
        t = case["tokens"]
        st["layer"] = layers.MoEMLP(case["hidden"], case["ffn"], case["experts"], case["topk"], t, None, gated=case["gated"], dtype=dt)
        with torch.no_grad():
            for p in st["layer"].parameters():
                p.copy_(mk.normal(*p.shape, std=0.02, dtype=p.dtype))
        st["x"] = mk.normal(t, case["hidden"], dtype=dt)
    elif kind == "route":
        st["chosen"], _ = mk.routing(case["tokens"], case["experts"], case["topk"])
        st["splits"] = torch.empty(case["experts"], dtype=torch.int32, device="cuda")
    else:
        raise ValueError(kind)
    return st


def run(st):
    kind = st["case"]["kind"]
    if kind == "gemm":
        return st["op"].forward(st["a"], st["b"], bias=st["bias"], input_scale=st["sa"], weight_scale=st["sb"])
    if kind == "mlp":
        y = st["ag"].forward(st["x"], st["w0"], bias=st["b0"])
        return y, st["rs"].forward(y, st["w1"], bias=st["b1"])
    if kind == "ag":
        return st["op"].forward(st["a"], st["b"], input_scale=st["sa"], weight_scale=st["sb"])
    if kind == "train":
        y = st["mlp"](st["x"])
        return (y.detach(),) + torch.autograd.grad(y, st["params"], st["dy"])
    if kind == "moe":
        y = st["l0"].forward(st["x"], st["w0"], st["splits"], st["si"], output_scale=st["scale0"])
        z = st["l1"].forward_gather_rs(y if st["act"] is None else st["act"], st["w1"], st["splits_cpu"], st["si"].view(-1),
                                       input_scale=st["in_scale"], weight_scale=st["scale1"], output_vec_scale=st["vec"])
        return y, z
    if kind == "layer":
        return st["layer"](st["x"])
    scatter_index, counts = flux.calc_scatter_index(st["chosen"], st["splits"], return_splits=True)
    return (scatter_index, counts) + tuple(flux.calc_gather_index(scatter_index))


def work(case):
    kind = case["kind"]
    size = 1 if case.get("dtype") in ("fp8", "int8") else 2
    if kind in ("gemm", "ag"):
        m, n, k = case["m"], case["n"], case["k"]
        full = case.get("bias") == "full"
        return {"bytes": (m + n) * k * size + (2 if full else 1) * m * n * 2, "flops": 2.0 * m * n * k}
    if kind == "mlp":
        m, h, f = case["m"], case["hidden"], case["ffn"]
        return {"bytes": 2 * h * f * 2 + (2 * m * h + m * f) * 2, "flops": 4.0 * m * h * f}
    if kind == "train":
        # six products; weights and activations in, output and all gradients out
        m, h, f = case["m"], case["hidden"], case["ffn"]
        return {"bytes": (4 * h * f + 4 * m * h) * 2, "flops": 12.0 * m * h * f}
    if kind in ("moe", "layer"):
        t, h, f, e, k = (case[x] for x in ("tokens", "hidden", "ffn", "experts", "topk"))
        gated = bool(case.get("gated"))
        used = e * (1.0 - (1.0 - k / e) ** t)  # experts that get at least one token, on average
        b = used * h * f * (3 if gated else 2) * size + t * h * (size + 2)
        if kind == "moe":
            b += t * k * f * 2 * (1 if size == 2 else 1.5)
        return {"bytes": b, "flops": (6.0 if gated else 4.0) * t * k * h * f}
    t, e, k = case["tokens"], case["experts"], case["topk"]
    return {"bytes": 4 * (t * k * 4 + e), "flops": 0.0}


# About four times what a pass differs from the same path in 64-bit arithmetic (2-norm, and the largest difference):
# one bf16 rounding gives 0.0017, a second product on top of it 0.0024, activations and gradients between 0.003 and
# 0.0042; fp16 an eighth of that. int8 products are whole numbers and their dequantisation is a fixed formula, and
# routing tables are integers: both are exact.
_TOLERANCE = {"gemm": (0.007, 0.016), "ag": (0.007, 0.016), "mlp": (0.01, 0.04), "moe": (0.012, 0.064), "train": (0.014, 0.072),
              "layer": (0.016, 0.072)}


def tolerance(case):
    if case["kind"] == "route" or case["dtype"] == "int8":
        return "exact"
    rel, most = _TOLERANCE[case["kind"]]
    if case["dtype"] == "fp16":
        return {"rel": rel / 8, "max": most / 8}
    return {"rel": rel, "max": most}


def _mm64(a, b):
    """a @ b.T in 64 bits, a block of b's rows at a time."""
    a = a.double()
    out = torch.empty((a.shape[0], b.shape[0]), dtype=torch.float64, device=a.device)
    for r in range(0, b.shape[0], 4096):
        out[:, r:r + 4096] = a @ b[r:r + 4096].double().t()
    return out


def _grouped64(rows, weights, splits):
    """Consecutive runs of `rows`, one per expert, each times its expert's weight."""
    return torch.cat([_mm64(part, weights[e]) for e, part in enumerate(torch.split(rows, splits))])


def _layer64(st):
    """A MoE layer from its definition: rows sorted by expert (ties in token order), weighted sum over the choices."""
    layer, x = st["layer"], st["x"]
    logits = x.double() @ layer.router.double().t()
    chosen = torch.topk(x.float() @ layer.router.t(), layer.topk, dim=1).indices  # which experts: a whole number
    w = torch.softmax(logits.gather(1, chosen), dim=1).reshape(-1)
    order = torch.argsort(chosen.reshape(-1), stable=True)
    splits = torch.bincount(chosen.reshape(-1), minlength=layer.nexperts).tolist()
    rows = x.double()[order // layer.topk]
    h = _grouped64(rows, layer.w_up, splits)
    if layer.w_gate is None:
        h = torch.nn.functional.gelu(h)
    else:
        h = torch.nn.functional.silu(_grouped64(rows, layer.w_gate, splits)) * h
    y = _grouped64(h, layer.w_down, splits) * w[order][:, None]
    return torch.zeros_like(x, dtype=torch.float64).index_add_(0, order // layer.topk, y)


def exact(case, seed):
    kind = case["kind"]
    if kind == "route":
        return None
    with torch.no_grad():
        st = prepare(case, seed)
        if kind in ("gemm", "ag"):
            out = _mm64(st["a"], st["b"].t() if case.get("weight_kn") else st["b"])
            if st["sa"] is not None:
                out *= st["sa"].double()[:, None] * st["sb"].double()[None, :]
            return out if st.get("bias") is None else out.add_(st["bias"])
        if kind == "mlp":
            y = _mm64(st["x"], st["w0"])
            y = y if st["b0"] is None else y.add_(st["b0"])
            z = _mm64(y, st["w1"])
            return y, (z if st["b1"] is None else z.add_(st["b1"]))
        if kind == "moe":
            splits = st["splits_cpu"].tolist()
            row_expert = torch.repeat_interleave(torch.arange(len(splits), device="cuda"), st["splits"].long())
            source = torch.empty(row_expert.numel(), dtype=torch.int64, device="cuda")
            source[st["si"].reshape(-1).long()] = torch.arange(source.numel(), device="cuda") // case["topk"]
            y = _grouped64(st["x"].double()[source], st["w0"], splits)
            if st["scale0"] is not None:
                y *= st["scale0"].double()[row_expert][:, None]
            z = _grouped64(y if st["act"] is None else st["act"], st["w1"], splits) * st["vec"].double()[:, None]
            if st["scale1"] is not None:
                z *= (st["in_scale"].double() * st["scale1"].double()[row_expert])[:, None]
            return y, torch.zeros((case["tokens"], z.shape[1]), dtype=torch.float64, device="cuda").index_add_(0, source, z)
        if kind == "layer":
            return _layer64(st)
    x = st["x"].detach().double().requires_grad_(True)
    params = [p.detach().double().requires_grad_(True) for p in st["mlp"].parameters()]
    w1, b1, w2, b2 = params if case["bias"] else (params[0], None, params[1], None)
    y = torch.nn.functional.linear(torch.nn.functional.gelu(torch.nn.functional.linear(x, w1, b1)), w2, b2)
    return (y.detach(),) + torch.autograd.grad(y, [x] + params, st["dy"].double())

"""Measured cases: the layers of a model that runs on this library, from one decode step to a long prefill.

Every case is the whole call chain a layer makes: the bf16 activation is quantised (or normalised and
quantised) and multiplied with a weight that was quantised when the model was loaded.  Sizes are those of
this repository's benchmark configurations and tests; ``draw`` spreads over the ranges between them.

kind        call chain
linear      group_wise_quant -> dense_gemm
norm        rms_norm_quant -> dense_gemm
lowlat      group_wise_quant (row-major scales) -> low_latency_mma_gemm
mlp         group_wise_quant -> dense_gemm(SituQuant) -> dense_gemm   (gate/up and down projection)
masked      group_wise_quant -> group_masked_gemm       (mixture of experts, fixed slots: decode)
contiguous  group_wise_quant -> group_contiguous_gemm   (mixture of experts, sorted rows: prefill)

``layers`` > 1 runs that many layers with activations and weights of their own, so that the weights come
from memory as they do in a model; ``graph`` replays them as one captured CUDA graph, as decode loops do.
"""

import math

import numpy as np
import torch

import halops_b200 as hq

MXFP8, MXFP4, NVFP4, W4A8 = "w8a8-mxfp8", "w4a4-mxfp4", "w4a4-nvfp4", "w4a8-mxfp4"

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def _case(name, kind, m, n, k, mode=MXFP8, dtype="bf16", tail=False, experts=1, layers=1, graph=False):
    c = dict(kind=kind, m=m, n=n, k=k, mode=mode, dtype=dtype, tail=tail, experts=experts, layers=layers, graph=graph)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: one small projection, latency and launches are all there is
        _case("linear-128x256x512", "linear", 128, 256, 512),
        # a decode step's projections for 8 sequences, weights from memory, heavy-tailed activations
        _case("decode-8x7168x2048-graph", "linear", 8, 7168, 2048, tail=True, layers=8, graph=True),
        # the same for 64 sequences and a wide projection
        _case("decode-64x24576x1536-graph", "linear", 64, 24576, 1536, tail=True, layers=4, graph=True),
        # latency-critical decode of 16 sequences through the entry point for row-major scales
        _case("lowlat-16x8192x4096-graph", "lowlat", 16, 8192, 4096, tail=True, layers=4, graph=True),
        # mixture of experts in decode: 20 experts with slots of 64 rows, partly filled
        _case("moe-masked-20x64x7168x2048", "masked", 64, 7168, 2048, experts=20),
        # a short prompt on a narrow projection
        _case("linear-512x1536x4096", "linear", 512, 1536, 4096),
        # a prompt of odd length in FP4, fp16 activations
        _case("linear-nvfp4-300x4096x4096", "linear", 300, 4096, 4096, mode=NVFP4, dtype="fp16"),
        # norm and projection of a prompt of 1000 tokens
        _case("norm-1000x8192x4096", "norm", 1000, 8192, 4096),
        # gated MLP block of a prefill of 4096 tokens (n: gate and up rows, the down projection is n/2 -> k)
        _case("mlp-4096x7168x2048", "mlp", 4096, 7168, 2048),
        # wide projection of a prefill in FP4
        _case("linear-nvfp4-4096x14336x4096", "linear", 4096, 14336, 4096, mode=NVFP4),
        # large square problem
        _case("linear-8192x8192x8192", "linear", 8192, 8192, 8192),
        # mixture of experts in prefill: 40960 rows sorted by expert, uneven runs
        _case("moe-contiguous-nvfp4-40960x4096x4096", "contiguous", 40960, 4096, 4096, mode=NVFP4, experts=10),
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of ``step`` in [lo, hi], evenly spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi, max(lo, round(v / step) * step)))


def draw(rng):
    while True:
        kind = rng.choice(["linear", "decode", "linear", "decode", "lowlat", "norm", "mlp", "masked", "contiguous"])
        mode = rng.choice([MXFP8, MXFP8, NVFP4, MXFP4])
        dtype = rng.choice(["bf16", "bf16", "fp16"])
        k_step, n_step = (128, 64) if mode == MXFP8 else (256, 128)
        if kind == "linear":
            c = _case("", kind, _log(rng, 65, 8192), _log(rng, 256, 16384, n_step), _log(rng, 512, 8192, k_step),
                      mode, dtype)
        elif kind == "decode":
            c = _case("", "linear", _log(rng, 1, 128), _log(rng, 1024, 24576, 64), _log(rng, 1024, 8192, 128),
                      tail=True, layers=rng.choice([4, 8]), graph=True)
        elif kind == "lowlat":
            c = _case("", kind, _log(rng, 1, 16), _log(rng, 1024, 24576, 8), _log(rng, 1024, 8192, 512),
                      tail=True, layers=rng.choice([4, 8]), graph=True)
        elif kind == "norm":
            c = _case("", kind, _log(rng, 65, 4096), _log(rng, 1024, 8192, 64), _log(rng, 1024, 8192, 128))
        elif kind == "mlp":
            c = _case("", kind, _log(rng, 65, 8192), _log(rng, 2048, 14336, 256), _log(rng, 1024, 4096, 128))
        elif kind == "masked":
            mode = rng.choice([MXFP8, W4A8, NVFP4])
            c = _case("", kind, rng.choice([64, 128, 256, 512]), _log(rng, 1024, 8192, 128),
                      _log(rng, 1024, 4096, 256), mode, experts=rng.randint(4, 24))
        else:
            mode = rng.choice([MXFP8, W4A8, NVFP4])
            c = _case("", kind, _log(rng, 1024, 40960, 64), _log(rng, 1024, 8192, 128), _log(rng, 1024, 4096, 256),
                      mode, experts=rng.randint(4, 20))
        w = work(c)
        # nothing above the large square problem
        if w["flops"] <= 2 * 8192**3 and w["bytes"] <= 1.5e9:
            return c


def _width(mode):
    """Bytes per element of the weight, elements per scale."""
    return {MXFP8: (1.0, 32), W4A8: (0.5, 32), MXFP4: (0.5, 32), NVFP4: (0.5, 16)}[mode]


def work(case):
    m, n, k, e, layers = (case[f] for f in ("m", "n", "k", "experts", "layers"))
    width, group = _width(case["mode"])
    rows = m
    if case["kind"] == "masked":
        rows = e * m // 2  # slots are half full on average; only valid rows are needed
    weights = e * n * k * (width + 1.0 / group)
    flops = 2.0 * rows * n * k
    out = 2.0 * rows * n
    if case["kind"] == "mlp":
        weights += (n // 2) * k * (width + 1.0 / group)
        flops += 2.0 * rows * (n // 2) * k
        out = 2.0 * rows * k
    return {"bytes": layers * (2.0 * rows * k + weights + out), "flops": layers * flops}


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32)


def _activation(case, g, rows):
    x = _normal(g, rows, case["k"])
    if case["tail"]:  # Student-t with 3 degrees of freedom: outliers as in a decoder's residual stream
        x = x / torch.sqrt((_normal(g, rows, case["k"]) ** 2 + _normal(g, rows, case["k"]) ** 2
                            + _normal(g, rows, case["k"]) ** 2) / 3.0)
    return x.clamp_(-6e4, 6e4).to(_DTYPES[case["dtype"]])


def _weight(g, n, k, mode, swizzle=True):
    w = (_normal(g, n, k) * 0.02).to(torch.bfloat16)
    return hq.group_wise_quant(w, MXFP4 if mode == W4A8 else mode, swizzle)


def _expert_weights(g, experts, n, k, mode):
    parts = [_weight(g, n, k, mode) for _ in range(experts)]
    return torch.stack([p[0] for p in parts]), torch.stack([p[1] for p in parts])


_capture_stream = []


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    kind, mode, m, n, k = (case[f] for f in ("kind", "mode", "m", "n", "k"))
    s = {"case": dict(case), "mode": mode, "quant_mode": MXFP8 if mode == W4A8 else mode}
    if kind in ("masked", "contiguous"):
        e = case["experts"]
        s["w"], s["sfw"] = _expert_weights(g, e, n, k, mode)
        s["alpha"] = 0.5 + torch.rand(e, generator=g, device="cuda") if mode == NVFP4 else None
        host = np.random.RandomState(seed % (1 << 32))
        if kind == "masked":
            s["x"] = _activation(case, g, e * m)
            s["rows"] = torch.from_numpy(host.randint(0, m + 1, e).astype(np.int32)).cuda()
            # rows that no token was routed to are not written: the buffer belongs to the program
            s["out"] = torch.zeros(e * m, n, dtype=torch.bfloat16, device="cuda")
        else:
            s["x"] = _activation(case, g, m)
            counts = host.multinomial(m // 64, host.dirichlet([8.0] * e)) * 64
            s["ids"] = torch.from_numpy(np.repeat(np.arange(e, dtype=np.int32), counts)).cuda()
        return s
    s["layers"] = []
    for _ in range(case["layers"]):
        x = _activation(case, g, m)
        if kind == "mlp":
            gate_up = hq.interleave_gate_up((_normal(g, n, k) * 0.02).to(torch.bfloat16))
            layer = (x, *hq.group_wise_quant(gate_up, mode), *_weight(g, k, n // 2, mode))
        elif kind == "norm":
            gamma = (1.0 + 0.1 * _normal(g, k)).to(torch.bfloat16)
            layer = (x, *_weight(g, n, k, mode), gamma)
        else:
            layer = (x, *_weight(g, n, k, mode, swizzle=kind != "lowlat"))
        s["layers"].append(layer)
    s["alpha"] = 0.5 + torch.rand(1, generator=g, device="cuda") if mode == NVFP4 else None
    if case["graph"]:
        # the decode loop's graph: captured once, replayed for every step
        if not _capture_stream:
            _capture_stream.append(torch.cuda.Stream())
        stream = _capture_stream[0]
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            _forward(s)
        torch.cuda.synchronize()
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"], stream=stream):
            s["out"] = _forward(s)
    return s


def _forward(s):
    kind, mode, n = s["case"]["kind"], s["mode"], s["case"]["n"]
    outs = []
    for layer in s["layers"]:
        x = layer[0]
        out = torch.empty(x.size(0), x.size(1) if kind == "mlp" else n, dtype=torch.bfloat16, device=x.device)
        if kind == "linear":
            q, sf = hq.group_wise_quant(x, mode)
            hq.dense_gemm(q, layer[1], sf, layer[2], out, alpha=s["alpha"], mode=mode)
        elif kind == "norm":
            q, sf = hq.rms_norm_quant(x, layer[3])
            hq.dense_gemm(q, layer[1], sf, layer[2], out, mode=mode)
        elif kind == "lowlat":
            q, sf = hq.group_wise_quant(x, mode, use_swizzle=False)
            hq.low_latency_mma_gemm(q, layer[1], sf, layer[2], out)
        else:
            q, sf = hq.group_wise_quant(x, mode)
            h = torch.empty(x.size(0), n // 2, dtype=torch.float8_e4m3fn, device=x.device)
            h_sf = torch.empty(sf.size(0), n // 64, dtype=torch.uint8, device=x.device)
            hq.dense_gemm(q, layer[1], sf, layer[2], h, mode=mode, epilogue=hq.EpilogueOp.SituQuant, output_sf=h_sf)
            hq.dense_gemm(h, layer[3], h_sf, layer[4], out, mode=mode)
        outs.append(out)
    return outs


def run(state):
    kind, mode = state["case"]["kind"], state["mode"]
    if "graph" in state:
        state["graph"].replay()
        return state["out"]
    if kind == "masked":
        q, sf = hq.group_wise_quant(state["x"], state["quant_mode"])
        hq.group_masked_gemm(q, state["w"], sf, state["sfw"], state["rows"], state["out"], alpha=state["alpha"],
                             max_m_per_expert=state["case"]["m"], mode=mode)
        return state["out"]
    if kind == "contiguous":
        x = state["x"]
        out = torch.empty(x.size(0), state["case"]["n"], dtype=torch.bfloat16, device=x.device)
        q, sf = hq.group_wise_quant(x, state["quant_mode"])
        hq.group_contiguous_gemm(q, state["w"], sf, state["sfw"], state["ids"], out, alpha=state["alpha"], mode=mode)
        return out
    return _forward(state)


def tolerance(case):
    # Against a float64 product of the same quantised operands, rounded to bf16, the results differ by a
    # rounding here and there: 2-norm up to 3.3e-5, largest value one bf16 step (7.7e-3); products with longer
    # K and other orders of the float32 sums show more such steps.  The gated MLP re-quantises its inner
    # activation to MXFP8 after approximate tanh: 5.8e-4 and 3.4e-2 against the float64 chain.
    return {"rel": 2.5e-3, "max": 0.14} if case["kind"] == "mlp" else {"rel": 5e-4, "max": 3e-2}

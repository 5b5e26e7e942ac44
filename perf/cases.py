"""The work that programs give this framework, as cases that can be timed and compared.

Five kinds, all through the entry points that a user's program calls:

  gemm    one ``skinny_gemm`` call, launched eagerly: the drop-in call of the torch op's users
  layers  the projections, norms and activations of consecutive decoder layers of a decode step
          (``residual_rms``, ``skinny_gemm``, ``llama_mlp_combined_ops``), captured once into a CUDA
          graph and replayed per step, as serving engines run decode
  mlp     one ``llama_mlp_combined_ops`` block, launched eagerly
  rms     one ``residual_rms`` call, eager       } decode rows up to prompt-processing rows, where the
  swiglu  one ``swiglu`` call, eager             } two element-wise kernels are used without the GEMM
  host    the projections of a decode step whose activations and results live in page-locked host
          memory (``HostBatch``: one library call a step), weights resident on the GPU

Attention is not part of the framework: its quantised output is an input of the o_proj call. Every
layer's hidden state is an input too, instead of the output of the layer before it: a rounding step
of a bf16 sum that lands on the other side of an fp8 boundary grows from layer to layer until two
correct results differ by percents, which would hide an incorrect one. Launches, their order and
what they read and write are the same.
Values: activations N(0, 1), weights N(0, 1/K) with a per-tensor e4m3 scale of amax / 448, so that
every projection's output is of order one. ``fnuz`` selects e4m3fnuz weights with fp16 activations
(the reference's types), otherwise e4m3fn with bf16.
"""
import math
import os
import sys

import torch

_PACKAGE_DIR = os.path.join(os.getcwd(), "hf-rocm-kernels_b200")
if _PACKAGE_DIR not in sys.path:
    sys.path.insert(1, _PACKAGE_DIR)

from hf_rocm_kernels import residual_rms, skinny_gemm, swiglu  # noqa: E402
from hf_rocm_kernels import _capi  # noqa: E402
from hf_rocm_kernels.combined_ops import llama_mlp_combined_ops  # noqa: E402

_EPS = 1e-5
_NORM_SCALE = 6.0 / 448    # the normalised activations stay below six
_ACT_SCALE = 12.0 / 448    # silu(gate) * up of order-one projections stays below twelve
_MAX_LAYER_BYTES = 850_000_000   # weights of one drawn state


def listed():
    return [
        # The smallest call there is: one token through a 4096 x 4096 projection, result allocated by
        # the call. Launches and latency are all that counts.
        {"name": "gemm_4096_m1", "kind": "gemm", "tokens": 1, "n": 4096, "k": 4096, "bias": False, "fnuz": False},
        # A ragged projection with bias: N no multiple of the tile, K no power of two, odd token count.
        {"name": "gemm_4104x5120_m13_bias", "kind": "gemm", "tokens": 13, "n": 4104, "k": 5120, "bias": True,
         "fnuz": False},
        # Decode of the Llama-3 8B projection shapes for a single user.
        {"name": "layers_8b_m1", "kind": "layers", "tokens": 1, "hidden": 4096, "qkv": 6144, "attn": 4096,
         "inter": 14336, "layers": 4, "fnuz": False},
        # The same for a batch of 16, the largest that the framework's benchmark runs.
        {"name": "layers_8b_m16", "kind": "layers", "tokens": 16, "hidden": 4096, "qkv": 6144, "attn": 4096,
         "inter": 14336, "layers": 4, "fnuz": False},
        # A batch of 64 with the reference's own types.
        {"name": "layers_8b_m64_fnuz", "kind": "layers", "tokens": 64, "hidden": 4096, "qkv": 6144, "attn": 4096,
         "inter": 14336, "layers": 4, "fnuz": True},
        # A server's full decode batch.
        {"name": "layers_8b_m256", "kind": "layers", "tokens": 256, "hidden": 4096, "qkv": 6144, "attn": 4096,
         "inter": 14336, "layers": 4, "fnuz": False},
        # The Llama-3 70B shapes on one GPU: the largest matrices.
        {"name": "layers_70b_m4", "kind": "layers", "tokens": 4, "hidden": 8192, "qkv": 10240, "attn": 8192,
         "inter": 28672, "layers": 2, "fnuz": False},
        # One rank's shards of the same under 8-way tensor parallelism (N split of qkv and gate/up, K
        # split of o_proj and down; the ranks' exchange is not part of it): many small matrices.
        {"name": "layers_70b_shard8_m16_fnuz", "kind": "layers", "tokens": 16, "hidden": 8192, "qkv": 1280,
         "attn": 1024, "inter": 3584, "layers": 4, "fnuz": True},
        # An MLP block outside a graph, ragged sizes.
        {"name": "mlp_5120x11008_m7", "kind": "mlp", "tokens": 7, "hidden": 5120, "inter": 11008, "fnuz": False},
        # Prompt processing: the two element-wise kernels at the rows of a prompt.
        {"name": "rms_4096x8192", "kind": "rms", "rows": 4096, "cols": 8192, "out": "fp8", "buffer": 0, "fnuz": False},
        {"name": "swiglu_2048x14336_fnuz", "kind": "swiglu", "rows": 2048, "hidden": 14336, "buffer": 0, "fnuz": True},
        # A decode step driven from host buffers.
        {"name": "host_8b_m16", "kind": "host", "tokens": 16, "hidden": 4096, "qkv": 6144, "attn": 4096,
         "inter": 14336, "layers": 4, "fnuz": False},
    ]


def _log_uniform(rng, low, high, step=1):
    """A multiple of ``step`` in [low, high], its logarithm uniform."""
    value = math.exp(rng.uniform(math.log(low), math.log(high)))
    return int(min(max(round(value / step), math.ceil(low / step)), high // step)) * step


def _dims(rng):
    """Dimensions of a decoder layer: a Llama-3 shape, one rank's shard of it, or a generic one."""
    pick = rng.random()
    if pick < 0.25:
        hidden, qkv, attn, inter = 4096, 6144, 4096, 14336
    elif pick < 0.5:
        hidden, qkv, attn, inter = 8192, 10240, 8192, 28672
    else:
        hidden = _log_uniform(rng, 1024, 8192, 16)
        attn = hidden
        qkv = hidden + 2 * _log_uniform(rng, max(64, hidden // 8), hidden, 8)
        inter = _log_uniform(rng, 2 * hidden, 7 * hidden // 2, 16)
    ways = rng.choice((1, 1, 1, 2, 4, 8))
    if ways > 1 and all(v % (16 * ways) == 0 for v in (qkv, attn, inter)):
        qkv, attn, inter = qkv // ways, attn // ways, inter // ways
    return {"hidden": hidden, "qkv": qkv, "attn": attn, "inter": inter}


def _layer_weight_bytes(c):
    return c["qkv"] * c["hidden"] + c["hidden"] * c["attn"] + 3 * c["inter"] * c["hidden"]


def draw(rng):
    kind = rng.choices(("gemm", "layers", "mlp", "rms", "swiglu", "host"), (5, 8, 2, 2, 2, 1))[0]
    fnuz = rng.random() < 0.4
    if kind == "gemm":
        return {"kind": kind, "tokens": _log_uniform(rng, 1, 256), "n": _log_uniform(rng, 1000, 28672),
                "k": _log_uniform(rng, 1024, 14336, 16), "bias": rng.random() < 0.4, "fnuz": fnuz}
    if kind == "rms":
        cols = _log_uniform(rng, 1024, 16384, rng.choice((1, 8, 8, 8, 128)))
        return {"kind": kind, "rows": _log_uniform(rng, 1, min(8192, 33_554_432 // cols)), "cols": cols,
                "out": rng.choice(("fp8", "fp8", "same")), "buffer": rng.choice((0, 0, 1024)), "fnuz": fnuz}
    if kind == "swiglu":
        hidden = _log_uniform(rng, 1000, 28672, rng.choice((1, 8, 8, 8, 128)))
        return {"kind": kind, "rows": _log_uniform(rng, 1, min(4096, 29_360_128 // hidden)), "hidden": hidden,
                "buffer": rng.choice((0, 0, 1024)), "fnuz": fnuz}
    c = {"kind": kind, "tokens": _log_uniform(rng, 1, 256 if kind != "host" else 64)}
    c.update(_dims(rng))
    if kind == "mlp":
        return {"kind": kind, "tokens": c["tokens"], "hidden": c["hidden"], "inter": c["inter"], "fnuz": fnuz}
    c.update(layers=max(1, min(4, _MAX_LAYER_BYTES // _layer_weight_bytes(c))), fnuz=fnuz)
    return c


# ------------------------------------------------------------------------------- preparation
class _Maker:
    """Seeded tensors on the GPU in the types of a case."""

    def __init__(self, case, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)
        self.fnuz = case["fnuz"]
        self.fp8 = torch.float8_e4m3fnuz if self.fnuz else torch.float8_e4m3fn
        self.act = torch.float16 if self.fnuz else torch.bfloat16

    def randn(self, *shape):
        return torch.randn(shape, generator=self.gen, device="cuda", dtype=self.act)

    def to_fp8(self, x, scale):
        """e4m3 bytes of ``x / scale`` and what a unit of them is worth (twice the scale as e4m3fnuz)."""
        q = (x * (1.0 / scale)).clamp_(-448.0, 448.0).to(torch.float8_e4m3fn)
        if not self.fnuz:
            return q, scale
        q = q.view(torch.int8)
        return torch.where(q == -128, 0, q).view(self.fp8), 2.0 * scale

    def weight(self, n, k):
        """Row-major [n, k] fp8 weight and its scale; values of N(0, 1/k) whose amax is taken as 5.5 sigma."""
        return self.to_fp8(self.randn(n, k), 5.5 / 448)[0], self.unit(5.5 / 448) / math.sqrt(k)

    def activation(self, m, k):
        return self.to_fp8(self.randn(m, k), 4.5 / 448)[0], self.unit(4.5 / 448)

    def unit(self, scale):
        return 2.0 * scale if self.fnuz else scale

    def scalar(self, value):
        return torch.tensor([value], dtype=torch.float32, device="cuda")


def _mlp_weights(make, hidden, inter):
    gate_up, s_gate_up = make.weight(2 * inter, hidden)
    down, s_down = make.weight(hidden, inter)
    return {"rms_weight": 1.0 + 0.1 * make.randn(hidden), "gate_up_weight": gate_up.t(),
            "gate_up_input_scale": make.scalar(make.unit(_NORM_SCALE)),
            "gate_up_output_scale": make.scalar(make.unit(_NORM_SCALE) * s_gate_up), "down_weight": down.t(),
            "down_input_scale": make.scalar(make.unit(_ACT_SCALE)),
            "down_output_scale": make.scalar(make.unit(_ACT_SCALE) * s_down)}


def _prepare_layers(case, make):
    tokens, hidden, qkv, attn, inter = (case[k] for k in ("tokens", "hidden", "qkv", "attn", "inter"))
    layers = []
    for _ in range(case["layers"]):
        w_qkv, s_qkv = make.weight(qkv, hidden)
        w_o, s_o = make.weight(hidden, attn)
        attn_out, s_attn = make.activation(tokens, attn)
        layers.append({
            "norm": 1.0 + 0.1 * make.randn(hidden), "norm_scale": make.scalar(make.unit(_NORM_SCALE)),
            "w_qkv": w_qkv.t(), "qkv_scale": make.scalar(make.unit(_NORM_SCALE) * s_qkv), "attn_out": attn_out,
            "w_o": w_o.t(), "o_scale": make.scalar(s_attn * s_o), "mlp": _mlp_weights(make, hidden, inter)})
    hidden_in = make.randn(case["layers"], tokens, hidden)
    residual_in = make.randn(case["layers"], tokens, hidden)

    def step():
        residuals = residual_in.clone()   # updated in place below
        outputs = []
        for w, x, residual in zip(layers, hidden_in, residuals):
            qkv_out = torch.empty((tokens, qkv), dtype=make.act, device="cuda")
            normed, residual = residual_rms(x, residual, w["norm"], _EPS, scale_tensor=w["norm_scale"],
                                            next_buffer=qkv_out, out_dtype=make.fp8)
            skinny_gemm(normed, w["w_qkv"], w["qkv_scale"], qkv_out)
            o_out = torch.zeros((tokens, hidden), dtype=make.act, device="cuda")
            skinny_gemm(w["attn_out"], w["w_o"], w["o_scale"], o_out)
            mlp_out, residual = llama_mlp_combined_ops(o_out, residual, rms_epsilon=_EPS, **w["mlp"])
            outputs.append({"qkv": qkv_out, "hidden": mlp_out, "residual": residual})
        return outputs

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outputs = step()
    return {"kind": "layers", "graph": graph, "outputs": outputs, "keep": (layers, hidden_in, residual_in)}


def _prepare_host(case, make):
    shapes = [(case["qkv"], case["hidden"], True), (case["hidden"], case["attn"], False),
              (2 * case["inter"], case["hidden"], False), (case["hidden"], case["inter"], False)] * case["layers"]
    m = case["tokens"]
    # all activations of the step in one page-locked block and all results in another
    a_block = torch.empty(sum(m * k for _, k, _ in shapes), dtype=torch.uint8).pin_memory()
    d_block = torch.zeros(sum(m * n for n, _, _ in shapes), dtype=make.act).pin_memory()
    calls, a_at, d_at = [], 0, 0
    for n, k, bias in shapes:
        w, s_w = make.weight(n, k)
        a, s_a = make.activation(m, k)
        a_host = a_block[a_at:a_at + m * k].view(make.fp8).view(m, k)
        d_host = d_block[d_at:d_at + m * n].view(m, n)
        a_host.view(torch.uint8).copy_(a.view(torch.uint8))
        call = (a_host, w, d_host, make.scalar(s_a * s_w), bias)
        if bias:
            d_in = (0.02 * make.randn(n)).repeat(m, 1).cpu().pin_memory()
            call += (d_in,)
        calls.append(call)
        a_at += m * k
        d_at += m * n
    batch = _capi.HostBatch(calls, torch.device("cuda", torch.cuda.current_device()))
    return {"kind": "host", "batch": batch, "stream": torch.cuda.Stream(), "outputs": [c[2] for c in calls],
            "keep": calls}


def prepare(case, seed):
    make = _Maker(case, seed)
    kind = case["kind"]
    if kind == "layers":
        return _prepare_layers(case, make)
    if kind == "host":
        return _prepare_host(case, make)
    if kind == "gemm":
        a, s_a = make.activation(case["tokens"], case["k"])
        w, s_w = make.weight(case["n"], case["k"])
        return {"kind": kind, "a": a, "b": w.t(), "scale": make.scalar(s_a * s_w),
                "bias": 0.02 * make.randn(1, case["n"]) if case["bias"] else None}
    if kind == "mlp":
        return {"kind": kind, "x": make.randn(case["tokens"], case["hidden"]),
                "residual": make.randn(case["tokens"], case["hidden"]),
                "weights": _mlp_weights(make, case["hidden"], case["inter"])}
    rows = case["rows"]
    buffer = torch.ones((rows, case["buffer"]), dtype=make.act, device="cuda") if case["buffer"] else None
    if kind == "rms":
        cols = case["cols"]
        return {"kind": kind, "x": make.randn(rows, cols), "residual": make.randn(rows, cols),
                "weight": 1.0 + 0.1 * make.randn(cols), "fp8": make.fp8, "buffer": buffer,
                "scale": make.scalar(make.unit(_NORM_SCALE)) if case["out"] == "fp8" else None}
    return {"kind": kind, "gate_up": make.randn(rows, 2 * case["hidden"]), "buffer": buffer,
            "scale": make.scalar(make.unit(_ACT_SCALE)), "fp8": make.fp8}


# ------------------------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "layers":
        state["graph"].replay()
        return state["outputs"]
    if kind == "gemm":
        a, bias = state["a"], state["bias"]
        # the call accumulates into the buffer it is given: the bias of every row, or a new one of zeros
        output = None if bias is None else bias.repeat(a.size(0), 1)
        return skinny_gemm(a, state["b"], state["scale"], output)
    if kind == "mlp":
        return llama_mlp_combined_ops(state["x"], state["residual"], rms_epsilon=_EPS, **state["weights"])
    if kind == "rms":
        outputs = residual_rms(state["x"], state["residual"], state["weight"], _EPS, scale_tensor=state["scale"],
                               next_buffer=state["buffer"], out_dtype=state["fp8"])
        return outputs if state["buffer"] is None or state["scale"] is None else (*outputs, state["buffer"])
    if kind == "swiglu":
        output = swiglu(state["gate_up"], state["scale"], next_buffer=state["buffer"], out_dtype=state["fp8"])
        return output if state["buffer"] is None else (output, state["buffer"])
    _capi.check(state["batch"].queue(state["stream"]))
    state["stream"].synchronize()
    return state["outputs"]


# ------------------------------------------------------------------------------- bytes and operations
def _gemm_work(m, n, k, bias=False):
    return n * k + m * k + 2 * m * n * (2 if bias else 1) + 4, 2 * m * n * k


def work(case):
    kind = case["kind"]
    if kind == "gemm":
        parts = [_gemm_work(case["tokens"], case["n"], case["k"], case["bias"])]
    elif kind == "rms":
        size = case["rows"] * case["cols"]
        parts = [(size * (6 + (1 if case["out"] == "fp8" else 2)) + 2 * case["cols"], 6 * size)]
        if case["out"] == "fp8":
            parts.append((2 * case["rows"] * case["buffer"], 0))
    elif kind == "swiglu":
        size = case["rows"] * case["hidden"]
        parts = [(5 * size + 2 * case["rows"] * case["buffer"], 6 * size)]
    else:
        # intermediate tensors need not reach memory: inputs, weights, returned tensors
        m, h, inter = case["tokens"], case["hidden"], case["inter"]
        mlp = [(3 * inter * h, 6 * m * inter * h)]
        if kind == "mlp":
            parts = mlp + [(2 * m * h * 4 + 2 * h, 0)]
        else:
            qkv, attn = case["qkv"], case["attn"]
            layer = mlp + [(qkv * h + 2 * m * qkv, 2 * m * qkv * h), (h * attn + m * attn, 2 * m * h * attn)]
            if kind == "host":   # every activation comes in and every result goes out
                layer += [(m * (2 * h + inter) + 2 * m * (qkv + 2 * h + 2 * inter), 0)]
            parts = layer * case["layers"] + ([(2 * m * h * 4 * case["layers"], 0)] if kind == "layers" else [])
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def tolerance(case):
    """About four times what another order of the fp32 sums (another K split) was seen to change.
    ``max`` covers one rounding step of the output type: 2^-8 .. 2^-7 of a 16-bit value, 1/8 of an fp8 one."""
    kind = case["kind"]
    if kind in ("gemm", "host"):     # single sums in another order: up to 7e-5 and one bf16 step
        return {"rel": 3e-4, "max": 2e-2}
    if kind in ("rms", "swiglu"):    # a few fp8 bytes per million on the other side of a boundary
        return {"rel": 5e-4, "max": 0.15}
    # several roundings to bf16 and fp8 in a row: up to 2.6e-3, largest single difference 5e-2
    return {"rel": 1e-2, "max": 0.15}


# ------------------------------------------------------------------------------- 64-bit results
def _matmul(a, w_nk, scale, bias=None):
    """scale * (a @ w^T) + bias in float64, a block of weight rows at a time."""
    a64, out = a.double(), []
    for rows in w_nk.cuda().split(8192):
        out.append(a64 @ rows.double().t())
    result = torch.cat(out, dim=1) * scale.double()
    return result if bias is None else result + bias.double()


def _quantise(y, fp8):
    """What an fp8 buffer holds of y; both formats saturate at the largest finite e4m3fn byte."""
    top = 224.0 if fp8 == torch.float8_e4m3fnuz else 448.0
    return y.clamp(-top, top), y.clamp(-top, top).float().to(fp8)


def _norm64(x, residual, weight):
    """The 16-bit sum that the norm reads, the sum before that rounding, the normalised rows."""
    exact_sum = x.double() + residual.double()
    s = exact_sum.to(x.dtype).double()
    return exact_sum, s * torch.rsqrt(s.square().mean(dim=1, keepdim=True) + _EPS) * weight.double()


def _swiglu64(gate_up, scale):
    gate, up = gate_up.double().chunk(2, dim=1)
    return torch.nn.functional.silu(gate) * up / scale.double()


def _mlp64(x, residual, w):
    fp8 = w["gate_up_weight"].dtype
    new_residual, y = _norm64(x, residual, w["rms_weight"])
    normed = _quantise(y / w["gate_up_input_scale"].double(), fp8)[1]
    gate_up = _matmul(normed, w["gate_up_weight"].t(), w["gate_up_output_scale"]).to(x.dtype)
    act = _quantise(_swiglu64(gate_up, w["down_input_scale"]), fp8)[1]
    return _matmul(act, w["down_weight"].t(), w["down_output_scale"]), new_residual


def exact(case, seed):
    """The outputs of ``run`` from torch in float64. Values that the operators hand on in 16 or 8 bits are
    rounded to them in between, as the operators define it; the returned ones are not rounded."""
    state = prepare(case, seed)
    kind = case["kind"]
    if kind == "gemm":
        return _matmul(state["a"], state["b"].t(), state["scale"], state["bias"])
    if kind == "mlp":
        return _mlp64(state["x"], state["residual"], state["weights"])
    if kind == "rms":
        new_residual, y = _norm64(state["x"], state["residual"], state["weight"])
        if state["scale"] is None:
            return y, new_residual
        y = _quantise(y / state["scale"].double(), state["fp8"])[0]
        return (y, new_residual) if state["buffer"] is None else (y, new_residual, torch.zeros_like(state["buffer"]))
    if kind == "swiglu":
        y = _quantise(_swiglu64(state["gate_up"], state["scale"]), state["fp8"])[0]
        return y if state["buffer"] is None else (y, torch.zeros_like(state["buffer"]))
    if kind == "host":
        results = []
        for call in state["keep"]:
            bias = call[5].cuda() if len(call) > 5 else None
            results.append(_matmul(call[0].cuda(), call[1], call[3], bias))
        return results
    layers, hidden_in, residual_in = state["keep"]
    results = []
    for w, x, residual in zip(layers, hidden_in, residual_in):
        new_residual, y = _norm64(x, residual, w["norm"])
        normed = _quantise(y / w["norm_scale"].double(), w["w_qkv"].dtype)[1]
        o_out = _matmul(w["attn_out"], w["w_o"].t(), w["o_scale"]).to(x.dtype)
        hidden, new_residual = _mlp64(o_out, new_residual.to(x.dtype), w["mlp"])
        results.append({"qkv": _matmul(normed, w["w_qkv"].t(), w["qkv_scale"]), "hidden": hidden,
                        "residual": new_residual})
    return results

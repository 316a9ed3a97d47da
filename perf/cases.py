"""The work that is timed: calls of the MoE block as a serving process makes them.

A case names one call on one layer.  Its fields:

    path    "block"       MoeBlock.forward: bf16 rows on the GPU in and out (the engine's resident path)
            "layer_step"  MoeBlock.layer_step: RMSNorm, block and residual add on the f32 residual stream
            "host_block"  MoeBlock.moe_ptr: bf16 rows in page-locked host memory in and out
            "experts"     backend.expert_group: the expert-layer call of the reference's engine, which
                          routes on the CPU and hands over f32 rows on the host, grouped by expert
    T       tokens of the call ("experts": most rows one expert gets; the counts are ragged)
    H, E, k, I, fmt, score, norm_topk, routed_scale, n_group, topk_group, shared
            the layer (fields of configs.MoeShape; `score` and `fmt` by name)
    bias_std, zipf   selection bias of a sigmoid router; Zipf exponent of the experts' popularity
    max_tokens       what the handle was created for: a server keeps one handle for decode and prefill

Weights, router, activations and row counts are made on the GPU from the seed alone; a state holds the
resident layer and its handle, as a program does that has loaded a model."""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from speedycolibri_b200 import backend
from speedycolibri_b200.configs import (CONFIGS, FMT_E4M3_ROW, FMT_FP8_B128, FMT_MXFP4, FMT_NVFP4, SCORE_SIGMOID,
                                        SCORE_SOFTMAX, MoeShape)
from speedycolibri_b200.moe import Config, Expert, Layer, MoeBlock

FORMATS = {"nvfp4": FMT_NVFP4, "mxfp4": FMT_MXFP4, "fp8_b128": FMT_FP8_B128, "e4m3_row": FMT_E4M3_ROW}
SCORES = {"softmax": SCORE_SOFTMAX, "sigmoid": SCORE_SIGMOID}
WEIGHT_STD = 0.02
MAX_WEIGHT_BYTES = 8.3e9   # the largest listed layer
MAX_FLOPS = 1.02e13        # the largest listed call
MAX_ROW_BYTES = 3.3e9      # and its rows


def _of_config(name: str, path: str, config: str, T: int, max_tokens: int, **other) -> dict:
    s = CONFIGS[config]
    case = dict(name=name, path=path, T=T, H=s.H, E=s.E, k=s.k, I=s.I,
                fmt=next(n for n, v in FORMATS.items() if v == s.fmt), score=next(n for n, v in SCORES.items() if v == s.score),
                norm_topk=s.norm_topk, routed_scale=s.routed_scale, n_group=s.n_group, topk_group=s.topk_group,
                shared=s.shared, bias_std=s.select_bias_std, zipf=s.zipf_s, max_tokens=max_tokens)
    case.update(other)
    return case


def listed() -> list[dict]:
    return [
        # decode of one conversation: launches and latency are what counts
        _of_config("decode_1", "block", "c1", 1, 2048),
        # a few conversations decoded together on the same layer
        _of_config("decode_8", "block", "c1", 8, 2048),
        # continuous batching on an FP8 layer, an odd number of live sequences
        _of_config("decode_fp8_21", "block", "c2", 21, 2048),
        # a full decode batch taken through the whole layer step around the block
        _of_config("decode_step_48", "layer_step", "c1", 48, 2048),
        # decode on a large layer: most of its experts are touched by a row or two each
        _of_config("decode_large_24", "block", "c3", 24, 4096),
        # the engine's own dispatch: routed on the CPU, f32 rows of 24 experts handed over from the host
        _of_config("experts_host", "experts", "c1", 12, 2048, E=24),
        # a short prompt on a small MXFP4 layer, an odd length
        _of_config("prompt_mxfp4_333", "block", "c0", 333, 2048, fmt="mxfp4"),
        # one prompt on an FP8 layer
        _of_config("prefill_fp8_512", "block", "c2", 512, 2048),
        # a prompt that comes from and goes back to host memory
        _of_config("prefill_host_1024", "host_block", "c1", 1024, 2048),
        # the ragged last chunk of a chunked prefill on a large layer
        _of_config("prefill_large_709", "block", "c3", 709, 4096),
        # a full prefill chunk on a large layer (the benchmark's headline call)
        _of_config("prefill_large_4096", "block", "c3", 4096, 4096),
        # many prompts at once with skewed expert popularity: the largest call
        _of_config("prefill_skewed_16384", "block", "c4", 16384, 16384),
    ]


def _log_uniform(rng: random.Random, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng: random.Random) -> dict:
    """A call of the same ranges: layers between c0's and c4's sizes, 1 to 16384 tokens, every format."""
    while True:
        path = rng.choice(["block", "block", "block", "block", "layer_step", "host_block", "experts"])
        H = int(_log_uniform(rng, 1024, 7168)) // 8 * 8
        I = int(_log_uniform(rng, 512, 2048)) // 8 * 8
        if rng.random() < 0.5:  # most real layers are multiples of 128; the rest only of 8
            H, I = H // 128 * 128, I // 128 * 128
        E = int(_log_uniform(rng, 32, 384))
        k = rng.randint(4, 8)
        sigmoid = rng.random() < 0.5
        groups = 8 if sigmoid and rng.random() < 0.5 else 1
        E = max(32, E // groups * groups)
        fmt = rng.choice(["nvfp4", "nvfp4", "fp8_b128", "e4m3_row", "mxfp4"])
        T = max(1, int(_log_uniform(rng, 1, 16400)))
        if path == "experts":
            E, T = rng.randint(1, 32), max(1, int(_log_uniform(rng, 1, 256)))
            k, groups = 1, 1
        case = dict(path=path, T=T, H=H, E=E, k=k, I=I, fmt=fmt, score="sigmoid" if sigmoid else "softmax",
                    norm_topk=rng.random() < 0.5, routed_scale=rng.choice([1.0, 2.5]), n_group=groups,
                    topk_group=4 if groups > 1 else 1, shared=path != "experts" and rng.random() < 0.7,
                    bias_std=0.01 if sigmoid else 0.0, zipf=0.0 if sigmoid else rng.choice([0.0, 0.6, 1.2]),
                    max_tokens=max(T, 2048))
        s = _shape(case)
        weights = (E + 1) * s.expert_bytes()
        rows = case["max_tokens"] * (k + 1) * H * 2
        if weights > MAX_WEIGHT_BYTES or rows > MAX_ROW_BYTES or work(case)["flops"] > MAX_FLOPS:
            continue
        if fmt == "mxfp4" and 3.0 * (E + 1) * H * I > 5e8:  # the container is transcoded on the host: small layers only
            continue
        return case


def _shape(case: dict) -> MoeShape:
    return MoeShape(str(case.get("name", "drawn")), H=case["H"], E=case["E"], k=case["k"], I=case["I"], T=case["T"],
                    fmt=FORMATS[case["fmt"]], score=SCORES[case["score"]], norm_topk=case["norm_topk"],
                    routed_scale=case["routed_scale"], n_group=case["n_group"], topk_group=case["topk_group"],
                    shared=case["shared"], select_bias_std=case["bias_std"], zipf_s=case["zipf"])


# ---- states -----------------------------------------------------------------------------------------
def _mxfp4(w: torch.Tensor):
    """f32 [O,K] on the GPU -> the container's host arrays: E2M1 nibbles and one E8M0 byte per 32."""
    O, K = w.shape
    nb = (K + 31) // 32
    blocks = torch.zeros((O, nb * 32), device=w.device)
    blocks[:, :K] = w
    blocks = blocks.view(O, nb, 32)
    exp = torch.floor(torch.log2(blocks.abs().amax(2).clamp_min(1e-30))) - 2.0
    scaled = blocks / torch.exp2(exp)[:, :, None]
    levels = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], device=w.device)
    code = torch.bucketize(scaled.abs().contiguous(), levels).to(torch.uint8) | (scaled < 0).to(torch.uint8) * 8
    code = code.view(O, nb * 32)[:, : (K + 1) // 2 * 2]
    nib = code[:, 0::2] | (code[:, 1::2] << 4)
    return nib.cpu().numpy(), (exp + 127.0).to(torch.uint8).cpu().numpy()


def _packed(fmt: int, O: int, K: int, gen: torch.Generator):
    """One matrix in its container's form: (codes, scales, tensor scale)."""
    w = torch.randn((O, K), generator=gen, device="cuda") * WEIGHT_STD
    if fmt == FMT_NVFP4:
        return backend.quantize_nvfp4_dev(w)
    if fmt == FMT_FP8_B128:
        return (*backend.quantize_fp8_b128_dev(w), 1.0)
    if fmt == FMT_E4M3_ROW:
        scales = w.abs().amax(1) / 448.0
        return (w / scales[:, None]).to(torch.float8_e4m3fn).view(torch.uint8), scales, 1.0
    return (*_mxfp4(w), 1.0)


def _matrix(fmt: int, O: int, K: int, gen: torch.Generator) -> backend.CudaTensor:
    codes, scales, g = _packed(fmt, O, K, gen)
    if fmt == FMT_MXFP4:
        return backend.CudaTensor.wrap_mxfp4(codes, scales, g, K, O)
    return backend.CudaTensor.from_device(fmt, codes, scales, g, K, O)


def _expert(s: MoeShape, gen: torch.Generator) -> Expert:
    return Expert(_matrix(s.fmt, s.I, s.H, gen), _matrix(s.fmt, s.I, s.H, gen), _matrix(s.fmt, s.H, s.I, gen))


def _host_rows(s: MoeShape, seed: int, gen: torch.Generator):
    # every seed has the same ragged counts, spread over the experts in another order
    rng = np.random.default_rng(seed)
    rows = [int(v) for v in rng.permutation(1 + np.random.default_rng(s.E).integers(0, s.T, s.E))]
    return rows, torch.randn((sum(rows), s.H), generator=gen, device="cuda").cpu().numpy()


def _router(s: MoeShape, seed: int, gen: torch.Generator):
    """(weights bf16 [E,H], selection bias or None, logit bias or None)"""
    rng = np.random.default_rng(seed)
    router = (torch.randn((s.E, s.H), generator=gen, device="cuda") / math.sqrt(s.H)).to(torch.bfloat16)
    popularity = -s.zipf_s * np.log(rng.permutation(s.E) + 1.0)
    return (router, (rng.standard_normal(s.E) * s.select_bias_std).astype(np.float32) if s.select_bias_std else None,
            (popularity - popularity.mean()).astype(np.float32) if s.zipf_s else None)


def _tokens(case: dict, s: MoeShape, gen: torch.Generator):
    """bf16 rows, or (f32 residual stream, norm weights) of a layer step"""
    x = torch.randn((s.T, s.H), generator=gen, device="cuda")
    if case["path"] == "layer_step":
        return x * 4.0, 1.0 + 0.1 * torch.randn(s.H, generator=gen, device="cuda")
    return x.to(torch.bfloat16)


def prepare(case: dict, seed: int) -> dict:
    backend.init([0])
    s = _shape(case)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    experts = [_expert(s, gen) for _ in range(s.E)]
    state = dict(path=case["path"], T=s.T)
    if case["path"] == "experts":
        rows, x = _host_rows(s, seed, gen)
        return dict(state, gates=[e.gate for e in experts], ups=[e.up for e in experts], downs=[e.down for e in experts],
                    rows=rows, x=x)
    router, select_bias, logit_bias = _router(s, seed, gen)
    layer = Layer(router=router.view(torch.int16).cpu().numpy().view(np.uint16), experts=experts, router_bias=select_bias,
                  logit_bias=logit_bias, shared=_expert(s, gen) if s.shared else None)
    state["block"] = MoeBlock(Config.from_shape(s), layer, case["max_tokens"])
    x = _tokens(case, s, gen)
    if case["path"] == "layer_step":
        return dict(state, resid=x[0], ln=x[1])
    if case["path"] == "host_block":
        return dict(state, x=x.cpu().pin_memory(), out=torch.empty((s.T, s.H), dtype=torch.bfloat16).pin_memory())
    return dict(state, x=x)


def run(state: dict):
    path = state["path"]
    if path == "block":
        return state["block"].forward(state["x"])
    if path == "layer_step":
        # the stream as attention leaves it; the step works in place on it
        return state["block"].layer_step(state["resid"].clone(), state["ln"], 1e-6)
    if path == "host_block":
        state["block"].moe_ptr(state["x"].data_ptr(), state["out"].data_ptr(), state["T"])
        return state["out"]
    return backend.expert_group(state["gates"], state["ups"], state["downs"], state["rows"], state["x"])


# ---- what the work cannot do without -------------------------------------------------------------------
def _active_experts(s: MoeShape) -> float:
    """Expected number of distinct routed experts of T tokens with k picks each."""
    p = (np.arange(s.E) + 1.0) ** -s.zipf_s
    return float(np.sum(1.0 - (1.0 - np.minimum(1.0, s.k * p / p.sum())) ** s.T))


def work(case: dict) -> dict:
    s = _shape(case)
    if case["path"] == "experts":
        rows = s.E * (s.T + 1) / 2.0
        return {"bytes": s.E * s.expert_bytes() + 8.0 * rows * s.H, "flops": 6.0 * s.H * s.I * rows}
    weights = (_active_experts(s) + (1 if s.shared else 0)) * s.expert_bytes() + 2.0 * s.E * s.H
    rows = (8.0 if case["path"] == "layer_step" else 4.0) * s.T * s.H
    return {"bytes": weights + rows, "flops": float(s.flops())}


def tolerance(case: dict) -> dict:
    # The result, h and the experts' rows are rounded to 16 bits.  Against the same arithmetic in 64 bits
    # the block measures 1.7e-3 to 2.9e-3 (largest difference 0.8e-2 to 1.5e-2 of the result's rms) over
    # these ranges; in the layer step the f32 residual stream carries most of the result's norm.
    if case["path"] == "layer_step":
        return {"rel": 4e-3, "max": 0.06}
    return {"rel": 1e-2, "max": 0.06}


# ---- the same results in 64 bits -------------------------------------------------------------------------
_E2M1 = [0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0, -0.0, -0.5, -1.0, -1.5, -2.0, -3.0, -4.0, -6.0]


def _dense(fmt: int, packed, O: int, K: int) -> torch.Tensor:
    """The f64 [O,K] weights that a packed matrix stands for."""
    codes, scales, g = packed
    if fmt in (FMT_FP8_B128, FMT_E4M3_ROW):
        w = codes.view(torch.float8_e4m3fn).double()
        if fmt == FMT_E4M3_ROW:
            return w * scales.double()[:, None]
        return w * scales.double().repeat_interleave(128, 0)[:O].repeat_interleave(128, 1)[:, :K]
    codes, scales = torch.as_tensor(codes, device="cuda").long(), torch.as_tensor(scales, device="cuda")
    table = torch.tensor(_E2M1, dtype=torch.float64, device="cuda")
    w = torch.stack((table[codes & 15], table[codes >> 4]), 2).reshape(O, -1)[:, :K]
    if fmt == FMT_NVFP4:
        return w * (scales.view(torch.float8_e4m3fn).double() * g).repeat_interleave(16, 1)[:, :K]
    return w * (torch.exp2(scales.double() - 127.0) * g).repeat_interleave(32, 1)[:, :K]


def _ffn(s: MoeShape, packed, x: torch.Tensor) -> torch.Tensor:
    gate, up, down = (_dense(s.fmt, m, *((s.H, s.I) if i == 2 else (s.I, s.H))) for i, m in enumerate(packed))
    return (torch.nn.functional.silu(x @ gate.T) * (x @ up.T)) @ down.T


def _route(s: MoeShape, x: torch.Tensor, router, select_bias, logit_bias):
    """(experts, weights) of every row: moe.rs:1047-1132 with the group limit and the logit bias"""
    z = x @ router.double().T
    if logit_bias is not None:
        z = z + torch.as_tensor(logit_bias, device="cuda").double()
    score = torch.sigmoid(z) if s.score == SCORE_SIGMOID else torch.softmax(z, 1)
    choice = score if select_bias is None else score + torch.as_tensor(select_bias, device="cuda").double()
    if s.n_group > 1:
        best = choice.view(s.T, s.n_group, -1).topk(2, dim=2).values.sum(2).topk(s.topk_group, dim=1).indices
        allowed = torch.zeros((s.T, s.n_group), dtype=torch.bool, device="cuda").scatter_(1, best, True)
        choice = choice.masked_fill(~allowed.repeat_interleave(s.E // s.n_group, 1), -math.inf)
    idx = choice.topk(s.k, dim=1).indices
    w = score.gather(1, idx)
    if s.norm_topk:
        w = w / w.sum(1, keepdim=True)
    return idx, w * s.routed_scale


def exact(case: dict, seed: int):
    backend.init([0])
    s = _shape(case)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    shapes = ((s.I, s.H), (s.I, s.H), (s.H, s.I))
    experts = [[_packed(s.fmt, O, K, gen) for O, K in shapes] for _ in range(s.E)]
    if case["path"] == "experts":
        rows, x = _host_rows(s, seed, gen)
        parts = torch.as_tensor(x, device="cuda").double().split(rows)
        return torch.cat([_ffn(s, e, part) for e, part in zip(experts, parts)]).cpu().numpy()
    routing = _router(s, seed, gen)
    shared = [_packed(s.fmt, O, K, gen) for O, K in shapes] if s.shared else None
    x = resid = _tokens(case, s, gen)
    if case["path"] == "layer_step":
        resid = x[0].double()
        normed = resid * torch.rsqrt(resid.pow(2).mean(1, keepdim=True) + 1e-6) * x[1].double()
        x = normed.to(torch.bfloat16)  # what the router and the experts are given
    x = x.double()
    idx, w = _route(s, x, *routing)
    out = _ffn(s, shared, x) if s.shared else torch.zeros_like(x)
    for e, packed in enumerate(experts):
        token, kk = (idx == e).nonzero(as_tuple=True)
        if len(token):
            out.index_add_(0, token, _ffn(s, packed, x[token]) * w[token, kk, None])
    if case["path"] == "layer_step":
        return out + resid
    return out.cpu() if case["path"] == "host_block" else out

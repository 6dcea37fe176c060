"""Performance cases of the MoE-FFN inference layer: what a user of the package runs.

Every case is ONE call of a public entry point (``MoeficationMoE.forward``, ``forward_block``,
``forward_host``) with the layer shapes of the benchmark's five model configurations and of the
parity fixtures, from a single image / a decode step to the largest prefill.  Weights are seeded
N(0, 0.02), inputs seeded N(0, 1) after the normalisation that stands in front of the layer.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import d2dmoe_b200 as D

DT = {"bf16": torch.bfloat16, "fp32": torch.float32}
ACT = {"relu": torch.nn.ReLU, "gelu": torch.nn.GELU}

# layer shapes: hidden width, expert width, experts, router width, activation, gated, input norm
SHAPES = {
    "vit": dict(d=768, H=128, E=24, R=128, act="relu", glu=False, norm="layer"),
    "gpt": dict(d=768, H=128, E=24, R=128, act="relu", glu=False, norm="layer"),
    "bert": dict(d=768, H=32, E=96, R=128, act="relu", glu=False, norm="layer"),
    "geglu": dict(d=2048, H=128, E=128, R=256, act="gelu", glu=True, norm="rms"),
    # a MoE-fied attention projection: narrow GELU experts, the layer adds its own input
    "proj": dict(d=768, H=32, E=12, R=128, act="gelu", glu=False, norm="layer"),
}


def _case(name, shape, B, S, dtype="bf16", mode="dynk_max", call="forward", tau_cfg=0.9, k=0):
    c = dict(shape=shape, B=B, S=S, dtype=dtype, mode=mode, call=call, tau_cfg=tau_cfg, k=k)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one 224x224 image through one layer: interactive classification, latency
        _case("vit_image", "vit", 1, 197),
        # one generation step of 32 sequences through a gated layer
        _case("geglu_decode_32", "geglu", 32, 1),
        # the fp32 layer of the reference's own CPU setting: 8 images
        _case("vit_fp32_8", "vit", 8, 197, dtype="fp32"),
        # an evaluation batch with the exact top-k gate
        _case("vit_topk_64", "vit", 64, 197, mode="topk", k=4),
        # a MoE-fied q/k/v/o projection of the same batch (residual inside the layer)
        _case("proj_residual_64", "proj", 64, 197),
        # half a transformer block on an odd batch, at a tau that keeps several experts
        _case("vit_block_37", "vit", 37, 197, call="block", tau_cfg=0.7),
        # router training: every expert on every token, output norms captured as labels
        _case("vit_labels_16", "vit", 16, 197, mode="all", call="labels"),
        # evaluation from host memory: pinned activations in, pinned activations out
        _case("vit_host_64", "vit", 64, 197, call="host"),
        # GPT-2 small, 32 x 1024 tokens, scores supplied by the caller's router
        _case("gpt2_scores_32k", "gpt", 32, 1024, call="scores"),
        # the headline evaluation batch
        _case("vit_256", "vit", 256, 197),
        # many small experts
        _case("bert_512", "bert", 512, 128),
        # the largest: prefill of 64 x 2048 tokens through a gated layer
        _case("geglu_prefill_128k", "geglu", 64, 2048),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["vit", "vit", "geglu", "geglu", "bert", "gpt", "proj", "fp32", "gate", "block",
                       "labels", "host"])
    tau = rng.choice([0.7, 0.8, 0.9, 0.95])
    if kind == "vit":
        return _case("", "vit", _log(rng, 1, 256), rng.choice([197, 50, 257]), tau_cfg=tau)
    if kind == "geglu":
        if rng.random() < 0.5:
            return _case("", "geglu", _log(rng, 1, 512), 1, tau_cfg=tau)
        return _case("", "geglu", rng.randint(1, 16), _log(rng, 16, 2048), tau_cfg=0.9)
    if kind == "bert":
        return _case("", "bert", _log(rng, 1, 512), rng.randint(16, 128), tau_cfg=0.9)
    if kind == "gpt":
        return _case("", "gpt", rng.randint(1, 32), _log(rng, 1, 1024), call="scores", tau_cfg=tau)
    if kind == "proj":
        return _case("", "proj", _log(rng, 1, 128), 197, tau_cfg=tau)
    if kind == "fp32":
        return _case("", "vit", _log(rng, 1, 32), rng.choice([197, 50]), dtype="fp32", tau_cfg=tau)
    if kind == "gate":
        mode = rng.choice(["topk", "dynk"])
        return _case("", "vit", _log(rng, 1, 128), 197, mode=mode, tau_cfg=rng.choice([0.2, 0.4]),
                     k=rng.randint(1, 8))
    if kind == "block":
        return _case("", "vit", _log(rng, 1, 256), 197, call="block", tau_cfg=tau)
    if kind == "labels":
        return _case("", "vit", _log(rng, 1, 64), 197, mode="all", call="labels")
    return _case("", "vit", _log(rng, 4, 128), 197, call="host", tau_cfg=tau)


class _GivenScores(torch.nn.Module):
    """A router of the user's own whose scores are already there."""

    def __init__(self, scores):
        super().__init__()
        self.scores = scores

    def forward(self, x):
        return self.scores


class State:
    pass


def prepare(case, seed):
    c, s = case, SHAPES[case["shape"]]
    dev, dt = torch.device("cuda"), DT[c["dtype"]]
    g = torch.Generator(device=dev).manual_seed(seed)

    def rn(*shape):
        return torch.randn(*shape, generator=g, device=dev)

    st = State()
    st.case = dict(c)
    x = rn(c["B"], c["S"], s["d"])
    if s["norm"] == "layer" and c["call"] != "block":      # the block call normalises itself
        x = torch.nn.functional.layer_norm(x, (s["d"],))
    elif s["norm"] == "rms":
        x *= torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6)
    st.x = x.to(dt)
    with torch.device(dev):
        m = D.MoeficationMoE("moe", s["d"], s["E"], not s["glu"], s["H"], ACT[s["act"]],
                             experts_class="execute_all" if s["glu"] else "custom_kernel",
                             add_residual_connection=c["shape"] == "proj",
                             add_intermediate_gating=s["glu"])
        m.router = D.MoeficationRouter(s["d"], s["E"], width=s["R"], depth=2, bias=False,
                                       activation="relu", output_activation="abs")
        norm = torch.nn.LayerNorm(s["d"], eps=1e-6)
    st.moe = m.to(dt).eval()
    st.norm = norm.to(dt)
    with torch.no_grad():
        for p in st.moe.parameters():
            p.copy_(rn(*p.shape) * 0.02)
        st.norm.weight.copy_(1.0 + 0.1 * rn(s["d"]))
        st.norm.bias.copy_(0.1 * rn(s["d"]))
    m.forward_mode, m.k, m.tau = c["mode"], c["k"], 1.0 - c["tau_cfg"]
    if c["mode"] == "dynk":
        m.tau = c["tau_cfg"]                 # cumulative share of the router's scores to cover
    if c["call"] == "scores":                # log-normal scores, as in the benchmark's GPT-2 layer
        m.router = _GivenScores(torch.exp(1.5 * rn(c["B"], c["S"], s["E"])).to(dt))
    if c["call"] == "labels":
        m.experts.capture_norms("output", 2)
    if c["call"] == "host":
        st.x = st.x.cpu().pin_memory()
        st.out = torch.empty_like(st.x).pin_memory()
    return st


def run(st):
    call = st.case["call"]
    if call == "host":
        return st.moe.forward_host(st.x, st.out)
    if call == "block":
        out, gating = st.moe.forward_block(st.x, st.norm)
    else:
        out, gating = st.moe(st.x)
    r = gating["moe"][0]
    # the 0/1 routing tensor as bit patterns: a decision is the same or it is not
    got = {"out": out, "routing": r.view(torch.int16 if r.element_size() == 2 else torch.int32)}
    if call == "labels":
        got["norms"] = st.moe.experts.captured_norms
    return got


_MEAN_K = {}


def _mean_k(c):
    """Expected number of experts a token keeps, from the distribution of its scores: the score
    of an expert is |N(0, 1)| up to a factor of the token's own, or log-normal where given."""
    s = SHAPES[c["shape"]]
    if c["mode"] == "all":
        return float(s["E"])
    if c["mode"] == "topk":
        return float(c["k"])
    key = (s["E"], c["call"] == "scores", c["mode"], c["tau_cfg"])
    if key not in _MEAN_K:
        z = np.random.RandomState(0).randn(4096, s["E"])
        z = np.exp(1.5 * z) if c["call"] == "scores" else np.abs(z)
        if c["mode"] == "dynk":
            p = -np.sort(-z / z.sum(1, keepdims=True), axis=1)
            kept = 1 + (np.cumsum(p, axis=1)[:, :-1] < c["tau_cfg"]).sum(1)
        else:
            kept = (z >= c["tau_cfg"] * z.max(1, keepdims=True)).sum(1)
        _MEAN_K[key] = float(kept.mean())
    return _MEAN_K[key]


def work(case):
    c, s = case, SHAPES[case["shape"]]
    n, es, G = c["B"] * c["S"], 4 if c["dtype"] == "fp32" else 2, 2 if s["glu"] else 1
    d, H, E, R = s["d"], s["H"], s["E"], s["R"]
    pairs = n * _mean_k(c)
    touched = E * (1.0 - (1.0 - pairs / (n * E)) ** n)       # experts that any token keeps
    flops = 2.0 * d * H * (G + 1) * pairs
    moved = 2.0 * n * d + touched * ((G + 1) * d * H + (0 if s["glu"] else H))
    if c["call"] == "scores":
        moved += n * E
    elif c["mode"] != "all":
        flops += 2.0 * n * (d * R + R * E)
        moved += d * R + R * E
    if c["call"] != "host":
        moved += n * E                                       # the routing tensor
    if c["call"] == "labels":
        moved += n * E
    return {"bytes": moved * es, "flops": flops}


def tolerance(case):
    # rel: fp32 sums / bf16 results with one rounding per added expert.  differ: a score that
    # lies within rounding of the threshold may fall on either side of it, where the layer
    # computes the scores itself.
    ties = case["mode"] != "all" and case["call"] != "scores"
    if case["dtype"] == "fp32":
        return {"rel": 1e-5, "differ": 1e-5 if ties else 0.0}
    return {"rel": 1e-2, "differ": 1e-4 if ties else 0.0}

"""The work a user of this package has it do, as cases that can be timed and compared.

A case is one MoE layer call the way an inference server issues it: router scores -> top-k -> ``fused_moe`` (kind
"layer"), or the preparation in front of a caller's own expert kernel, router -> ``moe_sorting`` -> 1x128 quantisation
(kind "prep"). Sizes are those of the benchmark configurations (DeepSeek-V3, Mixtral-8x7B and Qwen3-235B-A22B shaped
layers, the tiny layer) with batch sizes from one token to a long prefill; ``draw`` gives more of the same ranges, other
layer dimensions among them.

Fields of a case: M tokens, H model dim, I expert inner dim, E experts, local experts on this GPU (E unless experts are
sharded), topk; router "grouped" (sigmoid scores, group-limited) or "softmax"; skew "normal" (logits ~ N(0,1)) or "zipf"
(expert popularity follows Zipf(1.2)); quant "block" (1x128 / 128x128), "token" or "tensor"; x "bf16", "fp16" or "fp8"
(already quantised); act; live tokens (M unless the batch is padded); replay (the call is a captured graph).
"""

import math

import torch

import aiter_b200 as ab
from aiter_b200.graph import CapturedLayer

FP8 = torch.float8_e4m3fn
QUANT = {"block": ab.QuantType.per_1x128, "token": ab.QuantType.per_Token, "tensor": ab.QuantType.per_Tensor}
ACT = {"silu": ab.ActivationType.Silu, "gelu": ab.ActivationType.Gelu}
XTYPE = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp8": torch.bfloat16}
PREP_BLOCK = 32   # padding unit a caller's own kernel asks of moe_sorting (the default of that call)

DSV3 = dict(H=7168, I=2048, E=256, topk=8, router="grouped", skew="normal", quant="block")
QWEN3 = dict(H=4096, I=1536, E=128, topk=8, router="softmax", skew="zipf", quant="block")
MIXTRAL = dict(H=4096, I=14336, E=8, topk=2, router="softmax", skew="normal", quant="token")
TINY = dict(H=1024, I=512, E=8, topk=2, router="softmax", skew="normal", quant="tensor")


def _case(shape, M, kind="layer", local=None, x="bf16", act="silu", live=None, replay=False, **over):
    c = dict(kind=kind, M=M, **shape)
    c.update(over)
    c.update(local=c["E"] if local is None else local, x=x, act=act, live=M if live is None else live, replay=replay)
    return c


def listed():
    cases = {
        # one user's next token, Qwen3-shaped layer, launched from Python
        "token_m1": _case(QWEN3, 1),
        # a small decode batch whose layer call is captured once and replayed every step
        "decode_replay_m16": _case(QWEN3, 16, replay=True),
        # decode batch of the DeepSeek-V3-shaped layer (about half of the 256 experts are hit)
        "decode_dsv3_m64": _case(DSV3, 64),
        # a larger decode batch with skewed routing and an odd size
        "decode_zipf_m131": _case(QWEN3, 131),
        # decode of the Mixtral-shaped layer, row / channel scales
        "decode_mixtral_m32": _case(MIXTRAL, 32),
        # a chunk of a prefill mixed with decode tokens, fp16 model
        "mixed_zipf_m1000_fp16": _case(QWEN3, 1000, x="fp16"),
        # one rank of eight under expert parallelism: rows arrive quantised, the batch is padded
        "rank_dsv3_m2048_fp8": _case(DSV3, 2048, local=32, x="fp8", live=1777),
        # a small dense-ish layer, one scale per tensor, GELU
        "tiny_tensor_gelu_m513": _case(TINY, 513, act="gelu"),
        # prefill of the Mixtral-shaped layer
        "prefill_mixtral_m4096": _case(MIXTRAL, 4096),
        # a long prefill with skewed routing
        "prefill_zipf_m16384": _case(QWEN3, 16384),
        # the benchmark's prefill
        "prefill_dsv3_m8192": _case(DSV3, 8192),
        # what a caller with its own expert kernel needs of this package
        "prep_dsv3_m3001": _case(DSV3, 3001, kind="prep"),
    }
    return [dict(name=k, **v) for k, v in cases.items()]


def _flops(c):
    return 6.0 * c["live"] * c["topk"] * c["H"] * c["I"] * c["local"] / c["E"]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    biggest = listed()[10]
    most_flops, most_rows = _flops(biggest), biggest["M"] * biggest["topk"] * biggest["H"]
    family = rng.choice(["dsv3", "qwen3", "qwen3", "mixtral", "tiny", "other", "other", "rank", "prep"])
    shape = {"dsv3": DSV3, "qwen3": QWEN3, "mixtral": MIXTRAL, "tiny": TINY, "rank": DSV3, "prep": DSV3}.get(family)
    if shape is None:   # another layer of the same kind: any multiples of 128, any expert count
        H, I, E = 128 * _log_int(rng, 2, 64), 128 * _log_int(rng, 1, 32), _log_int(rng, 4, 256)
        while 3 * H * I * E > 11e9:
            E = max(4, E // 2)
        shape = dict(H=H, I=I, E=E, topk=rng.randint(1, min(8, E)), router="softmax", skew=rng.choice(["normal", "zipf"]),
                     quant=rng.choice(["block", "block", "token", "tensor"]))
    elif family == "mixtral":
        shape = dict(shape, quant=rng.choice(["token", "token", "tensor", "block"]))
    elif family == "tiny":
        shape = dict(shape, quant=rng.choice(["block", "token", "tensor"]))
    c = _case(shape, 1, kind="prep" if family == "prep" else "layer",
              x=rng.choice(["bf16", "bf16", "bf16", "fp16", "fp8"]), act=rng.choice(["silu", "silu", "silu", "gelu"]))
    if family == "rank":
        c["local"] = rng.choice([32, 64, 128])
    if family == "prep" and c["x"] == "fp8":
        c["x"] = "bf16"
    per_token = 6.0 * c["topk"] * c["H"] * c["I"] * c["local"] / c["E"]
    most = int(min(16384, 0.9 * most_flops / per_token, most_rows / (c["topk"] * c["H"])))
    c["M"] = c["live"] = _log_int(rng, 1, max(1, most))
    if family == "rank" and c["M"] > 8 and rng.random() < 0.5:
        c["live"] = rng.randint(c["M"] // 2, c["M"])
    c["replay"] = c["kind"] == "layer" and c["M"] <= 256 and rng.random() < 0.3
    return c


# ------------------------------------------------------------------------------------------ inputs
def _logits(c, g, device):
    """Router logits [M, E] fp32 and, for the grouped router, the correction bias. Zipf: log-popularity plus Gumbel noise,
    whose top-k is a draw without replacement from the popularity distribution."""
    M, E = c["M"], c["E"]
    bias = None
    if c["skew"] == "zipf":
        p = torch.arange(1, E + 1, dtype=torch.float32, device=device).pow(-1.2)
        u = torch.rand((M, E), generator=g, device=device).clamp_(1e-9, 1 - 1e-6)
        perm = torch.randperm(E, generator=g, device=device)
        logits = (p / p.sum()).log()[perm] - torch.log(-torch.log(u))
    else:
        logits = torch.randn((M, E), generator=g, device=device)
    if c["router"] == "grouped":
        bias = torch.randn((E,), generator=g, device=device) * 0.1
    return logits, bias


def _weights(E, N, K, quant, g, device):
    """[E, N, K] ~ N(0, 1/sqrt(K)) as e4m3 codes with scales amax/448 per 128x128 block, output channel or expert."""
    q = torch.empty((E, N, K), dtype=FP8, device=device)
    shape = {"block": (E, N // 128, K // 128), "token": (E, N, 1), "tensor": (E, 1)}[quant]
    s = torch.empty(shape, dtype=torch.float32, device=device)
    step = max(1, (1 << 26) // (N * K))
    for e in range(0, E, step):
        n = min(step, E - e)
        w = torch.randn((n, N, K), generator=g, device=device).mul_(1.0 / math.sqrt(K))
        v = w.view(n, N // 128, 128, K // 128, 128) if quant == "block" else w
        dims = {"block": (2, 4), "token": (2,), "tensor": (1, 2)}[quant]
        scale = v.abs().amax(dim=dims, keepdim=True) / 448.0
        q[e:e + n] = v.div_(scale).view(n, N, K).to(FP8)
        s[e:e + n] = scale.view(n, *shape[1:])
    return q, s


def prepare(case, seed):
    c = dict(case)
    dev = torch.device("cuda")
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    st = {"case": c}
    x = torch.randn((c["M"], c["H"]), generator=g, device=dev).to(XTYPE[c["x"]])
    logits, st["bias"] = _logits(c, g, dev)
    st["logits"] = logits if c["router"] == "grouped" else logits.to(torch.bfloat16)
    st["x"], st["a1_scale"] = x, None
    if c["kind"] == "prep":
        return st
    if c["x"] == "fp8":   # as the sender of an expert-parallel exchange quantised them
        st["x"], st["a1_scale"] = ab.get_hip_quant(QUANT[c["quant"]])(x, quant_dtype=FP8)
    st["w1"], st["w1_scale"] = _weights(c["local"], 2 * c["I"], c["H"], c["quant"], g, dev)
    st["w2"], st["w2_scale"] = _weights(c["local"], c["H"], c["I"], c["quant"], g, dev)
    st["mask"] = st["live"] = None
    if c["local"] < c["E"]:
        st["mask"] = torch.zeros(c["E"], dtype=torch.int32, device=dev)
        first = c["local"] * (seed % (c["E"] // c["local"]))
        st["mask"][first:first + c["local"]] = 1
    if c["live"] < c["M"]:
        st["live"] = torch.tensor([c["live"]], dtype=torch.int32, device=dev)
    if c["replay"]:
        st["layer"] = CapturedLayer(lambda x, logits: _layer(st, x, logits)[0], st["x"], st["logits"])
    return st


# ------------------------------------------------------------------------------------------ one pass
def _route(st, x, logits):
    c = st["case"]
    if c["router"] == "softmax":
        return ab.fused_topk(x, logits, c["topk"], True)
    w = torch.empty((c["M"], c["topk"]), dtype=torch.float32, device=logits.device)
    ids = torch.empty((c["M"], c["topk"]), dtype=torch.int32, device=logits.device)
    return ab.biased_grouped_topk(logits, st["bias"], w, ids, 8, 4, True, 2.5)


def _layer(st, x, logits):
    c = st["case"]
    w, ids = _route(st, x, logits)
    out = ab.fused_moe(x, st["w1"], st["w2"], w, ids, expert_mask=st["mask"], activation=ACT[c["act"]],
                       quant_type=QUANT[c["quant"]], w1_scale=st["w1_scale"], w2_scale=st["w2_scale"],
                       a1_scale=st["a1_scale"], num_local_tokens=st["live"])
    return out, w, ids


def run(state):
    c = state["case"]
    if c["kind"] == "prep":
        w, ids = _route(state, state["x"], state["logits"])
        routed = ab.moe_sorting(ids, w, c["E"], c["H"], XTYPE[c["x"]], PREP_BLOCK)
        return routed, ab.get_hip_quant(ab.QuantType.per_1x128)(state["x"], quant_dtype=FP8)
    if c["replay"]:
        return state["layer"](state["x"], state["logits"])
    return _layer(state, state["x"], state["logits"])


# ------------------------------------------------------------------------------------------ what a pass needs
def _active_experts(c):
    """Local experts that a batch of this case hits, from one seeded batch (all of them for a large one)."""
    g = torch.Generator()
    g.manual_seed(1)
    logits, bias = _logits(dict(c, M=min(c["live"], 1024)), g, "cpu")
    if c["router"] == "grouped":
        logits = logits.sigmoid() + bias
        groups = logits.view(logits.shape[0], 8, -1)
        kept = groups.topk(2, dim=-1)[0].sum(-1).topk(4, dim=-1)[1]
        keep = torch.zeros(groups.shape[:2]).scatter_(1, kept, 1.0)
        logits = (groups * keep[..., None]).flatten(1)
    ids = logits.topk(c["topk"], dim=-1)[1]
    return ids.unique().numel() * c["local"] / c["E"]


def work(case):
    c = dict(case)
    M, H, I, E, k = c["M"], c["H"], c["I"], c["E"], c["topk"]
    size = {"bf16": 2, "fp16": 2, "fp8": 1}[c["x"]]
    routing = M * E * (4 if c["router"] == "grouped" else 2) + 8.0 * M * k      # logits in, weights and ids out
    if c["kind"] == "prep":
        padded = M * k + E * PREP_BLOCK - k
        return {"bytes": routing + M * H * (size + 2 + 1 + 4.0 / 128) + 8.0 * padded, "flops": float(M * E)}
    scales = {"block": 3.0 * H * I / 16384, "token": 2.0 * I + H, "tensor": 2.0}[c["quant"]] * 4
    bytes_ = _active_experts(c) * (3.0 * H * I + scales) + routing + c["live"] * H * size + 2.0 * M * H
    return {"bytes": bytes_, "flops": max(1.0, _flops(c))}


def tolerance(case):
    if case["kind"] == "prep":
        return "exact"
    # bf16 / fp16 results; a rounding of the requantised activations that falls the other way moves single elements
    return {"rel": 1e-2, "max": 0.1}

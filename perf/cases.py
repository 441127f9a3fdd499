"""Performance cases: the pieces of a decomposition step that a user of this package runs, each through the entry
point a program calls, plus whole train steps.

A case is a dict with `path` (which piece), its sizes and its options. `listed()` holds the cases that are followed,
`draw(rng)` makes one more of the same ranges; `prepare` / `run` / `work` / `tolerance` / `exact` describe one case.
"""

from __future__ import annotations

import copy
import math

import torch
import torch.nn.functional as F

from param_decomp_b200.core.masking import SiteMask, StochasticSpec
from param_decomp_b200.ops.attention import flash_attention
from param_decomp_b200.ops.delta_rule import gated_delta_rule
from param_decomp_b200.ops.elementwise import squash_activity
from param_decomp_b200.ops.grouped import JobLayout, grouped_site
from param_decomp_b200.ops.site_linear import SiteWeights, fused_site_forward
from param_decomp_b200.ops.vocab_kl import kl_from_hidden, padded_logits

BF = torch.bfloat16
ALPHA = 0.01  # slope of the leaky sigmoids outside [0, 1]


def listed() -> list[dict]:
    return [
        # One site of the smoke-sized target (4 sequences of 128 tokens, 256 wide): the smallest masked forward and
        # backward a run makes, where launches and host time count.
        dict(name="site_small", path="site", tokens=512, d_in=256, C=256, d_out=256),
        # One attention site of the headline configuration (64 x 512 tokens, 768 -> 768, 4096 components), forward
        # and backward with a stochastic mask: 16 of these per draw and step.
        dict(name="site_768", path="site", tokens=32768, d_in=768, C=4096, d_out=768),
        # An MLP gate of the 8-billion-parameter shape (4096 -> 14336, 8192 components) on a ragged number of tokens.
        dict(name="site_8b_gate", path="site", tokens=3000, d_in=4096, C=8192, d_out=14336),
        # Causal self-attention of the headline target, forward and backward of a masked pass.
        dict(name="attn_512", path="attention", B=64, T=512, H=12, Hkv=12, hd=64, causal=True, segments=0, grad=True),
        # Grouped-query attention of the 8-billion-parameter shape at its sequence length.
        dict(name="attn_2048_gqa", path="attention", B=4, T=2048, H=32, Hkv=8, hd=128, causal=True, segments=0, grad=True),
        # Packed documents at an odd length (segmented rows), as the packed-row loader makes them.
        dict(name="attn_ragged", path="attention", B=4, T=777, H=8, Hkv=4, hd=64, causal=True, segments=3, grad=True),
        # Output loss of the headline target: KL over 50,277 logits of 16 sequences (a rank's share of
        # the batch on four GPUs), forward and backward to the hidden state.
        dict(name="kl_50k", path="vocab_kl", n=8192, V=50277, d=768),
        # Importance squash and minimality of one headline site, forward and backward.
        dict(name="squash_4096", path="squash", rows=32768, C=4096),
        # Gated DeltaNet recurrence of the hybrid target, forward and backward.
        dict(name="delta_128", path="delta", B=4, T=512, H=16, dk=128, dv=128),
        # Expert gate site of the mixture-of-experts configuration: 42 experts, top 8, 512 components each.
        dict(name="moe_gate", path="moe", tokens=8192, E=42, k=8, d=512, c=512, d_out=256),
        # Whole train step of the smoke configuration (host- and launch-bound).
        dict(name="step_small", path="step", layers=2, d_model=256, heads=4, d_ff=512, vocab=2000, C=256, batch=4, seq=128),
        # Whole train step at the headline widths on a small batch with fewer layers and components.
        dict(name="step_768", path="step", layers=2, d_model=768, heads=12, d_ff=3072, vocab=50277, C=1024, batch=8, seq=512),
    ]


def _log_int(rng, lo: int, hi: int, step: int = 1) -> int:
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng) -> dict:
    """One more case: sizes spread over the logarithm of the listed cases' ranges. Row counts and sequence lengths
    take any value; feature widths are multiples of 8 (the 16-byte rows every bf16 tensor of this package has)."""
    path = rng.choice(["site", "site", "attention", "attention", "vocab_kl", "squash", "delta", "moe"])
    if path == "site":
        while True:
            c = dict(path=path, tokens=_log_int(rng, 200, 32768), d_in=_log_int(rng, 128, 4096, 8),
                     C=_log_int(rng, 128, 8192, 8), d_out=_log_int(rng, 128, 14336, 8))
            if work(c)["flops"] <= 2.5e12:
                return c
    if path == "attention":
        while True:
            Hkv = rng.choice([1, 2, 4, 8, 12])
            c = dict(path=path, B=_log_int(rng, 1, 64), T=_log_int(rng, 100, 2048), H=Hkv * rng.choice([1, 1, 2, 4]),
                     Hkv=Hkv, hd=rng.choice([64, 64, 128, 128, 40, 96]), causal=rng.random() < 0.8,
                     segments=rng.choice([0, 0, 0, 3]), grad=rng.random() < 0.8)
            if work(c)["flops"] <= 4e11 and c["B"] * c["T"] * c["H"] <= 64 * 512 * 12:
                return c
    if path == "vocab_kl":
        while True:
            c = dict(path=path, n=_log_int(rng, 130, 8192), V=_log_int(rng, 2000, 151936), d=_log_int(rng, 256, 1024, 8))
            if c["n"] * c["V"] <= 8192 * 50277:
                return c
    if path == "squash":
        while True:
            c = dict(path=path, rows=_log_int(rng, 512, 65536), C=_log_int(rng, 128, 8192, 8))
            if c["rows"] * c["C"] <= 32768 * 4096:
                return c
    if path == "delta":
        while True:
            dk, dv = rng.choice([(128, 128), (128, 128), (64, 64), (64, 128), (32, 32)])
            c = dict(path=path, B=_log_int(rng, 1, 8), T=_log_int(rng, 60, 1024), H=_log_int(rng, 2, 32), dk=dk, dv=dv)
            if c["B"] * c["T"] * c["H"] <= 4 * 512 * 16:
                return c
    E = _log_int(rng, 4, 64)
    return dict(path="moe", tokens=_log_int(rng, 256, 8192), E=E, k=min(E, rng.choice([1, 2, 4, 8])),
                d=_log_int(rng, 128, 768, 64), c=_log_int(rng, 64, 512, 64), d_out=_log_int(rng, 128, 768, 64))


# ---- states -----------------------------------------------------------------------------------------------------


def _gen(seed: int, dev: str = "cuda") -> torch.Generator:
    return torch.Generator(device=dev).manual_seed(seed)


def _randn(g, *shape, scale: float = 1.0, dtype=BF) -> torch.Tensor:
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(dtype)


def _importances(g, *shape) -> torch.Tensor:
    """Lower-leaky importances: a clamp leaves many exact zeros, some exact ones and a spread between."""
    return (torch.randn(*shape, device="cuda", generator=g) * 0.6 + 0.2).clamp_(0, 1).to(BF)


def _segments(B: int, T: int, n: int) -> torch.Tensor:
    """`n` documents per row with boundaries that move from row to row."""
    cuts = torch.arange(T).repeat(B, 1) * n
    return ((cuts + torch.arange(B)[:, None] * (T // max(1, n * B))) // T).to(torch.int32).cuda()


def prepare(case: dict, seed: int):
    g, p = _gen(seed), case["path"]
    s = dict(case=case)
    if p == "site":
        n, di, C, do = case["tokens"], case["d_in"], case["C"], case["d_out"]
        V, U = _randn(g, di, C, scale=di**-0.5), _randn(g, C, do, scale=C**-0.5)
        s["w"] = SiteWeights(V, U, _randn(g, do, di, scale=di**-0.5), torch.zeros(di, C, device="cuda"),
                             torch.zeros(C, do, device="cuda"))
        s["x"] = _randn(g, n, di).requires_grad_(True)
        s["ci"] = _importances(g, n, C).requires_grad_(True)
        s["delta"] = torch.rand(n, 1, device="cuda", generator=g)
        s["spec"] = StochasticSpec(seed64=(seed << 32) | 9, stream=77, row_offset=0)
        s["dy"] = _randn(g, n, do)
    elif p == "attention":
        B, T, H, Hkv, hd = (case[k] for k in ("B", "T", "H", "Hkv", "hd"))
        s["qkv"] = [_randn(g, B, T, h, hd).requires_grad_(case["grad"]) for h in (H, Hkv, Hkv)]
        s["dy"] = _randn(g, B, T, H, hd)
        s["seg"] = _segments(B, T, case["segments"]) if case["segments"] else None
    elif p == "vocab_kl":
        n, V, d = case["n"], case["V"], case["d"]
        s["head"] = _randn(g, V, d, scale=1.5 * d**-0.5)
        hc = _randn(g, n, d)
        s["hm"] = (hc.float() + _randn(g, n, d, scale=0.3)).to(BF).requires_grad_(True)
        s["hc"] = hc
        s["clean"] = padded_logits(hc, s["head"])  # formed once per step and shared by its draws
        s["g"] = torch.ones((), device="cuda")
    elif p == "squash":
        s["pre"] = _randn(g, case["rows"], case["C"], scale=0.8).requires_grad_(True)
        s["dlower"] = _randn(g, case["rows"], case["C"])
        s["dact"] = torch.rand(case["C"], device="cuda", generator=g) * case["rows"]
    elif p == "delta":
        B, T, H, dk, dv = (case[k] for k in ("B", "T", "H", "dk", "dv"))
        q = F.normalize(torch.randn(B, T, H, dk, device="cuda", generator=g), dim=-1) * dk**-0.5
        k = F.normalize(torch.randn(B, T, H, dk, device="cuda", generator=g), dim=-1)
        v = torch.randn(B, T, H, dv, device="cuda", generator=g)
        gate = -F.softplus(torch.randn(B, T, H, device="cuda", generator=g) - 2)
        beta = torch.rand(B, T, H, device="cuda", generator=g)
        s["in"] = [t.requires_grad_(True) for t in (q, k, v, gate, beta)]
        s["dy"] = torch.randn(B, T, H, dv, device="cuda", generator=g)
    elif p == "moe":
        n, E, k, d, c, do = (case[x] for x in ("tokens", "E", "k", "d", "c", "d_out"))
        score = torch.randn(n, E, device="cuda", generator=g) + 0.5 * torch.randn(E, device="cuda", generator=g)
        top = score.topk(k, dim=-1)
        s["experts"], s["route_w"] = top.indices, torch.softmax(top.values, -1)
        s["V"], s["U"] = _randn(g, E, d, c, scale=d**-0.5), _randn(g, E, c, do, scale=c**-0.5)
        s["W"] = _randn(g, E, do, d, scale=d**-0.5)
        s["gV"], s["gU"] = torch.zeros(E, d, c, device="cuda"), torch.zeros(E, c, do, device="cuda")
        s["x"] = _randn(g, n, d).requires_grad_(True)
        s["mask"] = _importances(g, n * k, c).requires_grad_(True)
        s["delta"] = torch.rand(n * k, 1, device="cuda", generator=g)
        s["dy"] = _randn(g, n, do)
    else:
        s.update(_prepare_step(case, seed))
    return s


def _prepare_step(case: dict, seed: int) -> dict:
    from param_decomp_b200.config.experiments import LMExperimentConfig
    from param_decomp_b200.core.objective import build_objective
    from param_decomp_b200.core.recorded_step import RecordedTrainStep
    from param_decomp_b200.core.run import init_train_state
    from param_decomp_b200.core.train import StepContext
    from param_decomp_b200.experiments.lm.build import build_lm_run

    cfg = copy.deepcopy(_STEP_CONFIG)
    cfg["data"]["seq_len"] = case["seq"]
    cfg["data"]["train"]["seed"] = cfg["pd"]["seed"] = cfg["target"]["spec"]["seed"] = seed
    cfg["pd"]["batch_size"] = case["batch"]
    cfg["decomposition"]["sites"]["cs"] = {k: case["C"] for k in ("q", "k", "v", "o", "gate", "up", "down")}
    cfg["target"]["spec"]["arch"].update(n_layer=case["layers"], d_model=case["d_model"], n_head=case["heads"],
                                         d_ff=case["d_ff"], vocab_size=case["vocab"], max_seq_len=case["seq"])
    cfg = LMExperimentConfig.model_validate(cfg)
    dev = torch.device("cuda", torch.cuda.current_device())
    run_ = build_lm_run(cfg, None, dev)
    objective = build_objective(cfg.pd)
    ctx = StepContext.build(run_.model, objective, cfg.pd, lazy_masks=True)
    state = init_train_state(run_.model, run_.ci_fn, cfg.pd, objective, dev, case["batch"], case["seq"],
                             use_fused_optim=True)
    # the step API of a run: eager for its first calls, then recorded once and replayed
    return dict(step=RecordedTrainStep(ctx, state), state=state, batch=run_.sample_train(0))


_STEP_CONFIG = {
    "run_name": "perf",
    "cadence": {"checkpointing": {"kind": "none"}},
    "data": {"train": {"kind": "synthetic_zipf", "exponent": 1.1, "seed": 0},
             "eval": {"kind": "synthetic_zipf", "exponent": 1.1, "seed": 1}, "layout": "unsegmented_tokens", "seq_len": 128},
    "decomposition": {"sites": {"kind": "glu_transformer", "layers": {"kind": "all"}, "cs": {}},
                      "ci": {"type": "layerwise_mlp", "hidden_dims": [512]}},
    "pd": {
        "seed": 0, "batch_size": 4, "steps": 100000,
        "ci_fn_optimizer": {"lr_schedule": 1e-4, "grad_clip_norm": 1.0},
        "components_optimizer": {"lr_schedule": 1e-4, "grad_clip_norm": 1.0},
        "loss_metrics": [
            {"type": "ImportanceMinimalityLoss", "coeff": 1e-4, "gamma": 1.0},
            {"type": "StochasticReconLoss", "coeff": 1.0, "n_samples": 2},
            {"type": "FaithfulnessLoss", "coeff": 1000.0},
        ],
    },
    "runtime": {"mesh": {"replicate": 1, "fsdp": 1, "tp": 1}, "sharding": "ddp", "backend": "fused_sm100"},
    "target": {
        "spec": {"kind": "random_init", "seed": 0, "arch": {"family": "glu_transformer"}},
        "attention_implementation": "flash", "output_edge": {"kind": "materialized"}, "weights_dtype": "bfloat16",
    },
}


# ---- one pass ---------------------------------------------------------------------------------------------------


def run(s):
    case = s["case"]
    p = case["path"]
    if p == "site":
        w = s["w"]
        w.grad_V.zero_()  # the step's gradient buffers start from zero
        w.grad_U.zero_()
        y = fused_site_forward(s["x"], w, SiteMask(ci=s["ci"], delta=s["delta"], stochastic=s["spec"]), True)
        dx, dci = torch.autograd.grad(y, (s["x"], s["ci"]), s["dy"])
        return dict(y=y.detach(), dx=dx, dci=dci, dV=w.grad_V, dU=w.grad_U)
    if p == "attention":
        y = flash_attention(*s["qkv"], case["causal"], s["seg"])
        if not case["grad"]:
            return dict(y=y)
        dq, dk, dv = torch.autograd.grad(y, s["qkv"], s["dy"])
        return dict(y=y.detach(), dq=dq, dk=dk, dv=dv)
    if p == "vocab_kl":
        loss = kl_from_hidden(s["clean"], s["hm"], s["head"])
        (dh,) = torch.autograd.grad(loss, s["hm"], s["g"])
        return dict(loss=loss.detach(), dh=dh)
    if p == "squash":
        lower, act = squash_activity(s["pre"], 0.5, True, ALPHA)
        (dpre,) = torch.autograd.grad((lower, act), s["pre"], (s["dlower"], s["dact"]))
        return dict(lower=lower.detach(), act=act.detach(), dpre=dpre)
    if p == "delta":
        o = gated_delta_rule(*s["in"])
        return dict(o=o.detach(), grads=list(torch.autograd.grad(o, s["in"], s["dy"])))
    if p == "moe":
        k = case["k"]
        s["gV"].zero_()
        s["gU"].zero_()
        layout = JobLayout.build(s["experts"].reshape(-1), case["E"])
        y = grouped_site(layout.expand_tokens(s["x"], k), s["V"], s["U"], s["W"], layout, layout.scatter_rows(s["mask"]),
                         layout.scatter_rows(s["delta"])[:, 0].contiguous(), None, s["gV"], s["gU"], True)
        out = layout.combine(y, s["route_w"])
        dx, dm = torch.autograd.grad(out, (s["x"], s["mask"]), s["dy"])
        return dict(y=out.detach(), dx=dx, dm=dm, dV=s["gV"], dU=s["gU"])
    m = s["step"](s["batch"])
    return dict(losses={k: v for k, v in m.items() if k.startswith(("loss/", "grad_norm/"))},
                weights=[t.detach() for t in s["state"].components.parameters()])


# ---- what a pass cannot do without -------------------------------------------------------------------------------


def _pairs(case: dict) -> float:
    """(query, key) pairs of one head: documents are blocks of the attention matrix."""
    T, n = case["T"], max(1, case["segments"])
    return (T / n * (T / n + 1) / 2 if case["causal"] else (T / n) ** 2) * n


def work(case: dict) -> dict:
    p = case["path"]
    if p == "site":
        n, di, C, do = case["tokens"], case["d_in"], case["C"], case["d_out"]
        return dict(flops=2.0 * n * (3 * di * C + 3 * C * do + 2 * di * do),
                    bytes=2.0 * (2 * n * di + 2 * n * C + 2 * n * do + di * C + C * do + di * do) + 4.0 * (di * C + C * do))
    if p == "attention":
        B, T, H, Hkv, hd = (case[k] for k in ("B", "T", "H", "Hkv", "hd"))
        io = 2.0 * B * T * hd
        return dict(flops=(14.0 if case["grad"] else 4.0) * B * H * hd * _pairs(case),
                    bytes=io * (4 * H + 4 * Hkv) if case["grad"] else io * (2 * H + 2 * Hkv))
    if p == "vocab_kl":
        n, V, d = case["n"], case["V"], case["d"]
        return dict(flops=4.0 * n * V * d, bytes=2.0 * (n * V + 2 * n * d + V * d))
    if p == "squash":
        return dict(flops=0.0, bytes=8.0 * case["rows"] * case["C"] + 8.0 * case["C"])
    if p == "delta":
        B, T, H, dk, dv = (case[k] for k in ("B", "T", "H", "dk", "dv"))
        return dict(flops=18.0 * B * T * H * dk * dv, bytes=4.0 * B * T * H * (4 * dk + 4 * dv + 4))
    if p == "moe":
        n, E, k, d, c, do = (case[x] for x in ("tokens", "E", "k", "d", "c", "d_out"))
        return dict(flops=2.0 * n * k * (3 * d * c + 3 * c * do + 2 * d * do),
                    bytes=2.0 * (2 * n * d + 2 * n * do + 2 * n * k * c + E * (d * c + c * do + d * do)) + 4.0 * E * (d * c + c * do))
    L, d, ff, C, V = (case[x] for x in ("layers", "d_model", "d_ff", "C", "vocab"))
    n, h = case["batch"] * case["seq"], 512
    mats = [(d, d)] * 4 + [(d, ff)] * 2 + [(ff, d)]
    dense = L * sum(2.0 * n * i * o for i, o in mats)
    sites = L * sum(2.0 * n * (3 * i * C + 3 * C * o + 2 * i * o) for i, o in mats)
    ci = L * sum(6.0 * n * (i * h + h * C) for i, _ in mats)
    attn = L * case["batch"] * d * 2.0 * case["seq"] ** 2
    faith = L * sum(6.0 * i * C * o for i, o in mats)
    params = L * sum((i + o) * C + i * h + h * C for i, o in mats)
    return dict(flops=dense + 2 * sites + ci + attn * (1 + 2 * 3.5) + 2.0 * n * V * d * 5 + faith, bytes=28.0 * params)


# ---- how close another correct implementation comes ---------------------------------------------------------------


def tolerance(case: dict):
    return dict(rel=_TOLERANCE[case["path"]])


# Four times the distance from `exact` that a pass shows: bf16 outputs of bf16 products (site 2.4e-3, attention 2.7e-3,
# moe 3.3e-3, squash 1.7e-3), a difference of two softmaxes over bf16 logits (9.6e-3), 32-bit recurrences (3.2e-7, rounded
# up). A step's updated weights move by the sign of most gradients at first: a 1% change of a gradient flips under 1% of
# them (6e-4 of the weights), its losses are sums of bf16 quantities (1e-3).
_TOLERANCE = {"site": 1e-2, "attention": 1.1e-2, "vocab_kl": 4e-2, "squash": 7e-3, "delta": 2e-6, "moe": 1.3e-2, "step": 4e-3}


# ---- the same outputs in 64 bits ----------------------------------------------------------------------------------


def _philox_uniform(seed: int, stream: int, rows: int, cols: int) -> torch.Tensor:
    """The mask stream: Philox4x32 with 7 rounds over (column / 8, row, stream, 0x5044), 16 bits a value."""
    mask = 0xFFFFFFFF
    groups = (cols + 7) // 8
    c0 = torch.arange(groups, device="cuda")[None, :].expand(rows, groups)
    c1 = torch.arange(rows, device="cuda")[:, None].expand(rows, groups)
    c2, c3 = torch.full_like(c0, stream), torch.full_like(c0, 0x5044)
    k0, k1 = seed & mask, seed >> 32 & mask
    for _ in range(7):
        a, b = c0 * 0xD2511F53, c2 * 0xCD9E8D57
        c0, c1, c2, c3 = (b >> 32 & mask) ^ c1 ^ k0, b & mask, (a >> 32 & mask) ^ c3 ^ k1, a & mask
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    bits = torch.stack([h for w in (c0, c1, c2, c3) for h in (w & 0xFFFF, w >> 16)], -1).reshape(rows, groups * 8)
    return (bits[:, :cols].double() + 0.5) / 65536


def _site64(x, m, d, V, U, W, dy):
    """Masked site `((x V) * (m - d)) U + d (x W^T)` and its gradients."""
    H, co = x @ V, m - d
    A = H * co
    y = A @ U + d * (x @ W.T)
    dA = dy @ U.T
    dH = dA * co
    return y, dH @ V.T + (d * dy) @ W, dA * H, x.T @ dH, A.T @ dy


def exact(case: dict, seed: int):
    p = case["path"]
    if p == "step":
        return None
    s = prepare(case, seed)
    D = lambda t: t.detach().double()  # noqa: E731
    if p == "site":
        w, ci, d = s["w"], D(s["ci"]), D(s["delta"])
        u = _philox_uniform(s["spec"].seed64, 77, *ci.shape)
        y, dx, dm, dV, dU = _site64(D(s["x"]), ci + (1 - ci) * u, d, D(w.V), D(w.U), D(w.W), D(s["dy"]))
        return dict(y=y, dx=dx, dci=dm * (1 - u), dV=dV, dU=dU)
    if p == "attention":
        outs = [_attention64(case, *(D(t[b]) for t in s["qkv"]), D(s["dy"][b]), None if s["seg"] is None else s["seg"][b])
                for b in range(case["B"])]
        return {k: torch.stack([o[k] for o in outs]) for k in outs[0]}
    if p == "vocab_kl":
        head, n, tot, dh = D(s["head"]), case["n"], 0.0, []
        for i in range(0, n, 2048):
            lc, lm = (torch.log_softmax(D(h[i:i + 2048]) @ head.T, -1) for h in (s["hc"], s["hm"]))
            pc = lc.exp()
            tot = tot + (pc * (lc - lm)).sum()
            dh.append((lm.exp() - pc) @ head / n)
        return dict(loss=tot / n, dh=torch.cat(dh))
    if p == "squash":
        x, g, rows, g2 = D(s["pre"]), D(s["dlower"]), case["rows"], 0.25
        u = torch.where(x > 1, 1 + ALPHA * (x - 1), x.clamp(0, 1))
        du = torch.where(x > 1, ALPHA, (x > 0).double())
        dl = torch.where(x > 1, 0.0, torch.where(x > 0, g, ALPHA * g.clamp(max=0)))
        act = ((1 + g2) * u * u / (u * u + g2)).mean(0)
        return dict(lower=x.clamp(0, 1), act=act, dpre=dl + D(s["dact"]) / rows * (1 + g2) * 2 * u * g2 / (u * u + g2) ** 2 * du)
    if p == "delta":
        leaves = [D(t).requires_grad_(True) for t in s["in"]]
        o = _delta64(*leaves)
        return dict(o=o.detach(), grads=list(torch.autograd.grad(o, leaves, D(s["dy"]))))
    E, k = case["E"], case["k"]
    x, mask, d, dy, rw = D(s["x"]), D(s["mask"]), D(s["delta"]), D(s["dy"]), D(s["route_w"])
    V, U, W = D(s["V"]), D(s["U"]), D(s["W"])
    out = dict(y=torch.zeros_like(dy), dx=torch.zeros_like(x), dm=torch.zeros_like(mask), dV=torch.zeros_like(V), dU=torch.zeros_like(U))
    flat, w_flat = s["experts"].reshape(-1), rw.reshape(-1)
    for e in range(E):
        j = (flat == e).nonzero()[:, 0]
        t, w = j // k, w_flat[j][:, None]
        y, dx, dm, out["dV"][e], out["dU"][e] = _site64(x[t], mask[j], d[j], V[e], U[e], W[e], dy[t] * w)
        out["y"].index_add_(0, t, y * w)
        out["dx"].index_add_(0, t, dx)
        out["dm"][j] = dm
    return out


def _attention64(case: dict, q, k, v, dy, seg):
    T, group = case["T"], case["H"] // case["Hkv"]
    keep = torch.ones(T, T, dtype=torch.bool, device=q.device)
    if case["causal"]:
        keep = keep.tril()
    if seg is not None:
        keep = keep & (seg[:, None] == seg[None, :])
    scale = case["hd"] ** -0.5
    q, k, v, dy = (t.transpose(0, 1) for t in (q, k, v, dy))  # [heads, T, hd]
    kr, vr = k.repeat_interleave(group, 0), v.repeat_interleave(group, 0)
    P = torch.softmax((q @ kr.transpose(1, 2) * scale).masked_fill(~keep, float("-inf")), -1)
    y = P @ vr
    if not case["grad"]:
        return dict(y=y.transpose(0, 1))
    dP = dy @ vr.transpose(1, 2)
    dS = P * (dP - (dy * y).sum(-1, keepdim=True)) * scale
    fold = lambda t: t.reshape(case["Hkv"], group, T, -1).sum(1).transpose(0, 1)  # noqa: E731
    return dict(y=y.transpose(0, 1), dq=(dS @ kr).transpose(0, 1), dk=fold(dS.transpose(1, 2) @ q), dv=fold(P.transpose(1, 2) @ dy))


def _delta64(q, k, v, g, beta):
    """Token-by-token recurrence; 64-token spans are recomputed in the backward pass to bound its memory."""
    from torch.utils.checkpoint import checkpoint

    def span(S, q, k, v, g, beta):
        outs = []
        for t in range(q.shape[1]):
            S = S * g[:, t].exp()[..., None, None]
            delta = (v[:, t] - torch.einsum("bhij,bhi->bhj", S, k[:, t])) * beta[:, t][..., None]
            S = S + k[:, t][..., :, None] * delta[..., None, :]
            outs.append(torch.einsum("bhij,bhi->bhj", S, q[:, t]))
        return S, torch.stack(outs, 1)

    B, T, H, dk = q.shape
    S = q.new_zeros(B, H, dk, v.shape[-1])
    outs = []
    for t in range(0, T, 64):
        S, o = checkpoint(span, S, *(a[:, t:t + 64] for a in (q, k, v, g, beta)), use_reentrant=False)
        outs.append(o)
    return torch.cat(outs, 1)

"""What this framework is used for, as measurable cases: training passes, optimizer updates, whole optimizer steps and
evaluation passes of the model families of ``autoresearch_b200.config`` through the entry points that a training
program calls (``GPT``, ``ParamLayout``, ``MuonAdamW``, ``Trainer``), on one GPU.

Kinds of a case:

* ``train``: one micro-step as every trainer runs it: main gradients cleared, forward, backward into the fp32 main
  gradients.  Returned: the per-token losses and every gradient.
* ``eval``: the scoring pass of the bits-per-byte evaluation, no gradients.  Returned: the per-token losses (the model
  hands out no logits).
* ``optim``: one Muon + AdamW update of all parameters from given gradients.  Returned: parameters, fp32 masters and
  moments.
* ``step``: ``Trainer.train_step()``: batch staging, gradient accumulation, schedule, optimizer.  Returned: the loss,
  the gradients and the updated parameters.

Weights are drawn on the GPU in the engine's initial distributions, except that the matrices the initialisation sets to
zero (output projections, gates, router) get small values, as they have after the first steps: no product is
trivially zero.  Tokens are Zipf(1.1) distributed, as in the synthetic stream of the trainers.
"""
from __future__ import annotations

import math

import torch

from autoresearch_b200.config import ModelConfig, MoEConfig, ScheduleConfig, TrainConfig
from autoresearch_b200.models.gpt import GPT
from autoresearch_b200.ops.backend import get_backend
from autoresearch_b200.optim.muon_adamw import MuonAdamW
from autoresearch_b200.parallel.layout import ParamLayout
from autoresearch_b200.trainer import Trainer

HEAD = 128
MID_RUN = 400          # optimizer steps that the state of an optimizer has behind it
DEVICE = "cuda"


def _case(name, kind, d_model, layers, batch, seq, vocab=8192, experts=0, capacity=1.25, accum=1):
    c = dict(kind=kind, d_model=d_model, layers=layers, batch=batch, seq=seq, vocab=vocab, experts=experts,
             capacity=capacity, accum=accum)
    return dict(c, name=name) if name else c


def listed():
    return [
        # --- the smallest calls: the `small` preset of the tests and the smoke run.  Launches and host time count.
        _case("eval small, 1 x 512", "eval", 256, 4, 1, 512, vocab=1024),
        _case("train small, 2 x 512", "train", 256, 4, 2, 512, vocab=1024),
        # a whole optimizer step of the same model, two accumulated micro-steps: what a first trial run does
        _case("step small, 2 x 2 x 512", "step", 256, 4, 2, 512, vocab=1024, accum=2),
        # --- the 119.5 M model (phase 1), 30 layers of 512: one sequence (debugging, small memory) ...
        _case("train 119M, 1 x 2048", "train", 512, 30, 1, 2048),
        # ... and the 64 sequences per micro-step its recipe trains with
        _case("train 119M, 64 x 2048", "train", 512, 30, 64, 2048),
        # --- odd and ragged: three heads, a sequence that ends inside a tile, a vocabulary that is no power of two
        _case("train odd, 5 x 1531", "train", 384, 12, 5, 1531, vocab=5000),
        # --- the 428 M model (phase 2) at its full context of 32768 tokens: training and scoring
        _case("train 428M, 1 x 32768", "train", 1024, 30, 1, 32768),
        _case("eval 428M, 1 x 32768", "eval", 1024, 30, 1, 32768),
        # --- the mixture-of-experts model (8 experts, top 2, capacity factor 1.25) at its context of 8192, the four
        #     sequences per micro-step of the benchmark
        _case("train MoE 2.2B, 4 x 8192", "train", 1024, 30, 4, 8192, experts=8),
        # --- the wide model (1.6 B, 16 heads) at its context of 8192
        _case("train wide 1.6B, 1 x 8192", "train", 2048, 30, 1, 8192),
        # --- the optimizer alone, which every step ends with
        _case("optim 119M", "optim", 512, 30, 1, 2048),
        _case("optim 428M", "optim", 1024, 30, 1, 32768),
    ]


# ------------------------------------------------------------------------------------------------
def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """Widths of 1 to 16 heads, 2 to 30 layers, sequences of 128 to 32768 tokens (half of them no multiple of anything),
    batches that keep a pass within the cost and the memory of the largest listed ones."""
    top = max(work(c)["flops"] for c in listed())
    while True:
        kind = rng.choice(["train", "train", "train", "eval", "eval", "step", "optim"])
        heads = rng.choice([1, 2, 2, 3, 4, 4, 5, 6, 8, 8, 12, 16])
        layers = rng.choice([2, 3, 4, 6, 8, 12, 18, 24, 30])
        vocab = rng.choice([1024, 2048, 4096, 5000, 6144, 8192, 8192])
        experts, capacity = 0, 1.25
        if kind in ("train", "eval") and rng.random() < 0.2:
            experts, capacity = rng.choice([4, 8]), rng.choice([1.25, 2.0])
            if kind == "train" and (heads < 8 or layers < 18):
                # one token that goes to another expert on a near tie shows in single gradient elements of a small
                # model; scored losses hardly move
                kind = "eval"
        seq = int(_log_uniform(rng, 128, 32768))
        if rng.random() < 0.5:
            seq = max(128, seq // 128 * 128)
        batch = max(1, int(_log_uniform(rng, seq, 131072) // seq))
        accum = 1
        if kind == "step":
            # Trainer draws its weights on the host: models of a size at which that stays short
            heads, layers = min(heads, 4), min(layers, 12)
            accum = rng.choice([1, 2, 3, 4])
            batch = max(1, min(batch, 32768 // seq))
        c = _case(None, kind, heads * HEAD, layers, batch, seq, vocab, experts, capacity, accum)
        n = _model_config(c).num_params()["total"]
        # what a backward pass keeps, per token and layer: 12 D values, with experts their gathered rows as well
        act = 2.0 * c["d_model"] * (14 + (10 * 2 * capacity if experts else 0)) * batch * seq
        kept = act * (layers if kind in ("train", "step") else 2)
        if work(c)["flops"] <= top and kept <= 50e9 and n <= 1.7e9 and not (kind == "optim" and n > 4.5e8):
            return c


# ------------------------------------------------------------------------------------------------
def _model_config(case):
    D = case["d_model"]
    moe = None
    if case["experts"]:
        moe = MoEConfig(n_experts=case["experts"], top_k=2, mlp_dim_e=4 * D, capacity_factor=case["capacity"])
    return ModelConfig(vocab=case["vocab"], seq_len=case["seq"], d_model=D, n_head=D // HEAD, head_dim=HEAD,
                       mlp_dim=4 * D, n_layer=case["layers"], moe=moe, name="case")


def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _draw_moments(opt, layout, g):
    """Optimizer state in the middle of a run, as after loading a checkpoint (the first Adam steps from zero moments
    would be plus or minus the learning rate, whatever the gradient)."""
    for gi, st in opt.state.items():
        st["master"].copy_(layout.group_view(layout.flat_param, layout.groups[gi]))
        if "momentum" in st:
            st["momentum"].normal_(0.0, 1e-4, generator=g)
            st["second"].uniform_(0.5, 1.5, generator=g).div_(max(layout.groups[gi].shape))
        else:
            st["m"].normal_(0.0, 1e-5, generator=g)
            st["v"].uniform_(1e-8, 4e-8, generator=g)


@torch.no_grad()
def _draw_weights(model, g):
    cfg = model.cfg
    s = cfg.init_scale * math.sqrt(3.0) / math.sqrt(cfg.d_model)
    for name, p, kind in model.named_matrix_groups():
        leaf = name.split(".")[-1]
        if leaf == "wte":
            p.normal_(0.0, 1.0, generator=g)
        elif leaf in ("lm_head", "router"):
            p.normal_(0.0, 0.02, generator=g)
        elif leaf == "resid_lambdas":
            p.fill_(1.0)
        elif leaf == "x0_lambdas":
            p.fill_(0.1)
        elif leaf in ("wo", "wdn", "expert_proj", "ve_gate"):
            p.uniform_(-0.25 * s, 0.25 * s, generator=g)
        else:
            p.uniform_(-s, s, generator=g)


def _tokens(case, g, seed):
    """ids and targets [batch, seq] int32, Zipf(1.1) over a shuffled vocabulary."""
    B, T, V = case["batch"], case["seq"], case["vocab"]
    w = torch.arange(1, V + 1, device=DEVICE, dtype=torch.float64).pow_(-1.1)
    cdf = torch.cumsum(w, 0) / w.sum()
    u = torch.rand(B, T + 1, generator=g, device=DEVICE, dtype=torch.float64)
    rank = torch.searchsorted(cdf, u).clamp_(max=V - 1)
    tok = torch.randperm(V, generator=g, device=DEVICE)[rank].to(torch.int32)
    ids, targets = torch.empty(B, T, device=DEVICE, dtype=torch.int32), torch.empty(B, T, device=DEVICE, dtype=torch.int32)
    # staging buffers that a training loop refills in place: some batches have passed through them already
    for _ in range(1 + int(seed) % 61):
        ids.copy_(tok[:, :-1])
        targets.copy_(tok[:, 1:])
    return ids, targets


def prepare(case, seed):
    cfg = _model_config(case)
    kind = case["kind"]
    if kind == "step":
        tokens = case["batch"] * case["seq"] * case["accum"]
        tcfg = TrainConfig(device_batch_size=case["batch"], total_batch_size=tokens, max_steps=1000, cooldown_steps=300,
                           synthetic_data=True, synthetic_kind="zipf", impl="sm100", cooldown_trigger_file="",
                           seed=int(seed) % (1 << 31), schedule_cfg=ScheduleConfig(peak_lr=0.02))
        tr = Trainer(cfg, tcfg, device=DEVICE, quiet=True)
        with torch.no_grad():
            _draw_weights(tr.model, _generator(seed))
            _draw_moments(tr.opt, tr.layout, _generator(seed + 1))
        tr.step = MID_RUN
        return dict(kind=kind, trainer=tr)
    g = _generator(seed)
    model = GPT(cfg, get_backend("sm100", cfg), dtype=torch.bfloat16, device=DEVICE)
    _draw_weights(model, g)
    if kind == "eval":
        ids, targets = _tokens(case, g, seed)
        return dict(kind=kind, model=model, ids=ids, targets=targets)
    layout = ParamLayout(model.named_matrix_groups())
    if kind == "train":
        ids, targets = _tokens(case, g, seed)
        return dict(kind=kind, model=model, layout=layout, ids=ids, targets=targets,
                    scale=1.0 / (case["batch"] * case["seq"]))
    opt = MuonAdamW(layout, ScheduleConfig(peak_lr=0.02), cfg.d_model, kernels=model.backend.optim_kernels())
    for grp in layout.groups:
        # matrices: a decaying spectrum of row scales over noise, the shape that summed token gradients have
        v = layout.group_view(layout.flat_grad, grp)
        v.normal_(0.0, 1e-4, generator=g)
        if v.dim() == 3:
            v.mul_(torch.logspace(0.0, -1.0, v.shape[1], device=DEVICE)[None, :, None])
    with torch.no_grad():
        _draw_moments(opt, layout, g)
    return dict(kind=kind, model=model, layout=layout, opt=opt, step=MID_RUN)


def run(state):
    kind = state["kind"]
    if kind == "step":
        tr = state["trainer"]
        loss = tr.train_step()
        return dict(loss=loss, grad=tr.layout.flat_grad, param=tr.layout.flat_param)
    model = state["model"]
    if kind == "eval":
        with torch.no_grad():
            _, per_token = model(state["ids"], state["targets"])
        return dict(per_token=per_token)
    layout = state["layout"]
    if kind == "train":
        layout.zero_grad()
        scaled, per_token = model(state["ids"], state["targets"], grad_scale=state["scale"])
        scaled.backward()
        layout.accumulate_autograd_grads()
        return dict(per_token=per_token, grad=layout.flat_grad)
    opt = state["opt"]
    state["step"] += 1
    opt.step(state["step"], 0.0)
    return dict(param=layout.flat_param, state=[[st[k] for k in sorted(st)] for st in opt.state.values()])


# ------------------------------------------------------------------------------------------------
def _forward_flops(case):
    """Multiply-adds times two of one forward pass: matrices of every token, attention over the keys a query sees."""
    cfg = _model_config(case)
    B, T, D, V = case["batch"], case["seq"], case["d_model"], case["vocab"]
    n = B * T
    mlp = 8 * D * D * (2 if case["experts"] else 1) + case["experts"] * D       # top 2 of the experts and the router
    flops = 2.0 * n * (V * D + cfg.n_layer * (4 * D * D + mlp))
    for l in range(cfg.n_layer):
        w = min(cfg.window(l), T)
        keys = T * (T + 1) / 2 if w >= T else (w + 1) * (w + 2) / 2 + (T - w - 1) * (w + 1)
        flops += 4.0 * B * D * keys
    return flops


def _optimizer_work(case):
    cfg = _model_config(case)
    D, L, M = case["d_model"], cfg.n_layer, 4 * case["d_model"]
    p = cfg.num_params()
    mats = [(4 * L, D, D)] + ([(case["experts"] * L, M, D), (case["experts"] * L, D, M)] if case["experts"] else [(L, M, D), (L, D, M)])
    muon = sum(c * m * n for c, m, n in mats)
    # Newton-Schulz: five times Gram matrix (symmetric: half), its square (symmetric: half), product
    flops = sum(5.0 * c * (m * n * min(m, n) + min(m, n) ** 3 + 2.0 * m * n * min(m, n)) for c, m, n in mats)
    # fp32 gradient and bf16 parameter; fp32 master and one (Muon) or two (AdamW) moments are read and written
    return muon * (4 + 2 + 16) + (p["total"] - muon) * (4 + 2 + 24), flops


def work(case):
    cfg = _model_config(case)
    p = cfg.num_params()["total"]
    n = case["batch"] * case["seq"]
    fwd = _forward_flops(case)
    if case["kind"] == "eval":
        return {"bytes": 2 * p + 12 * n, "flops": fwd}
    if case["kind"] == "train":
        return {"bytes": 2 * p + 4 * p + 12 * n, "flops": 3 * fwd}
    b, f = _optimizer_work(case)
    if case["kind"] == "optim":
        return {"bytes": b, "flops": f}
    return {"bytes": case["accum"] * (2 * p + 4 * p + 12 * n) + b, "flops": case["accum"] * 3 * fwd + f}


def tolerance(case):
    """About four times what other correct orders of the same bf16 arithmetic give: 1-CTA instead of 2-CTA GEMM tiles,
    64-wide instead of 128-wide attention tiles, RoPE and norms as separate kernels instead of GEMM epilogues; for the
    optimizer the library path.  Seen, relative in the 2-norm (largest element): gradients 3e-4 to 2.3e-3 (0.03 to 0.4,
    single small elements), losses 4e-4 (0.002), updated parameters 7e-4 (0.03).  With experts a token on a near tie
    may be routed differently: gradients 0.009 (1.8 of 2e9 elements), losses 1e-3 (0.02)."""
    if case["kind"] == "eval":
        return {"rel": 0.004, "max": 0.08} if case["experts"] else {"rel": 0.0016, "max": 0.01}
    if case["kind"] == "optim":
        return {"rel": 0.004, "max": 0.08}
    return {"rel": 0.03, "max": 0.99} if case["experts"] else {"rel": 0.01, "max": 0.99}

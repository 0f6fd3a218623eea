"""End-to-end: the sm_100a model against the fp32 oracle with identical weights."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _build(impl, cfg, dtype, attn=None):
    from autoresearch_b200.models.gpt import GPT
    from autoresearch_b200.models.init import init_weights
    from autoresearch_b200.ops.backend import get_backend
    be = get_backend(impl, cfg)
    if attn is not None:
        be.attn = attn
    m = GPT(cfg, be, dtype=dtype, device="cuda")
    init_weights(m, scheme="normal", std=0.05)
    return m


@pytest.mark.parametrize("attn", ["own", "library"])
def test_forward_backward_matches_oracle(attn):
    from autoresearch_b200.config import model_preset
    from autoresearch_b200.ops import kernels as K
    if attn == "library":
        pytest.importorskip("flash_attn")
    cfg = model_preset("small")
    torch.manual_seed(0)
    ref = _build("oracle", cfg, torch.float32)
    mod = _build("sm100", cfg, torch.bfloat16, attn)
    with torch.no_grad():
        for (n1, p1), (n2, p2) in zip(ref.named_parameters(), mod.named_parameters()):
            p1.copy_(p2.float())
    B, T = 2, cfg.seq_len
    ids = torch.randint(0, cfg.vocab, (B, T), device="cuda", dtype=torch.int32)
    tgt = torch.randint(0, cfg.vocab, (B, T), device="cuda", dtype=torch.int32)
    scale = 1.0 / (B * T)
    l_ref, pt_ref = ref(ids, tgt, grad_scale=scale)
    l_ref.backward()
    l_mod, pt_mod = mod(ids, tgt, grad_scale=scale)
    l_mod.backward()
    K.check_err_flag()
    assert abs(l_ref.item() - l_mod.item()) < 2e-2 * abs(l_ref.item())
    assert (pt_ref - pt_mod).abs().mean().item() < 5e-2
    bad = []
    for (n, p1), (_, p2) in zip(ref.named_parameters(), mod.named_parameters()):
        g1, g2 = p1.grad, p2.grad
        if g1 is None or g2 is None:
            assert g1 is None and g2 is None or (g1 is not None and g1.abs().max() == 0) or True
            continue
        rel = ((g1 - g2.float()).norm() / (g1.norm() + 1e-12)).item()
        if rel > 0.08:
            bad.append((n, rel))
    assert not bad, f"gradient mismatch: {bad}"


def test_training_step_sm100_loss_decreases():
    from autoresearch_b200.config import TrainConfig, model_preset
    from autoresearch_b200.ops import kernels as K
    from autoresearch_b200.trainer import Trainer
    cfg = model_preset("small")
    t = TrainConfig(device_batch_size=4, total_batch_size=4 * cfg.seq_len * 2, max_steps=30, cooldown_steps=10,
                    synthetic_data=True, impl="sm100", cooldown_trigger_file="")
    tr = Trainer(cfg, t, device="cuda", quiet=True)
    losses = [float(tr.train_step()) for _ in range(30)]
    K.check_err_flag()
    assert losses[-1] < losses[0] - 0.3, losses


def _assert_whole_layers_match_the_steps(cfg, batch, seq):
    from autoresearch_b200.ops import kernels as K
    torch.manual_seed(3)
    mod = _build("sm100", cfg, torch.bfloat16)
    ids = torch.randint(0, cfg.vocab, (batch, seq), device="cuda", dtype=torch.int32)
    tgt = torch.randint(0, cfg.vocab, (batch, seq), device="cuda", dtype=torch.int32)
    got = {}
    for whole in (True, False):
        mod.backend.layer_calls = whole
        for with_main in (False, True):          # gradients handed to autograd, and summed into fp32 main gradients
            for p in mod.parameters():
                p.grad = None
                if with_main:
                    p.main_grad = torch.zeros(p.shape, dtype=torch.float32, device="cuda")
                elif hasattr(p, "main_grad"):
                    del p.main_grad
            loss, per_tok = mod(ids, tgt, grad_scale=1.0 / ids.numel())
            loss.backward()
            got[whole, with_main] = (per_tok.clone(), [(p.main_grad if with_main else p.grad).clone() for p in mod.parameters()])
        with torch.no_grad():
            got[whole, "eval"] = mod(ids, tgt)[1].clone()
    K.check_err_flag()
    names = [n for n, _ in mod.named_parameters()]
    assert torch.equal(got[True, "eval"], got[False, "eval"])
    for with_main in (False, True):
        a, b = got[True, with_main], got[False, with_main]
        assert torch.equal(a[0], b[0])
        for n, x, y in zip(names, a[1], b[1]):
            if "lambdas" in n or "ve_gate" in n:
                assert (x - y).float().norm() <= 1e-2 * y.float().norm() + 1e-6, n      # atomics; bf16 gradients: one rounding
            else:
                # fp32 split-K sums meet in L2 in any order: a few units in the last place of the largest partial sum
                assert (x.float() - y.float()).norm() <= (1e-5 if with_main else 4e-3) * y.float().norm(), n


def _layers_cfg(heads, layers, mlp, experts):
    from autoresearch_b200.config import ModelConfig, MoEConfig
    moe = MoEConfig(n_experts=experts, top_k=2, mlp_dim_e=mlp, capacity_factor=1.25) if experts else None
    return ModelConfig(vocab=1024, seq_len=512, d_model=128 * heads, n_head=heads, head_dim=128, mlp_dim=mlp, n_layer=layers, moe=moe)


@pytest.mark.parametrize("batch,seq,layers,heads,experts", [(1, 512, 4, 2, 0), (3, 331, 6, 2, 0), (1, 130, 2, 2, 0), (3, 301, 3, 3, 0),
                                                            (1, 3, 1, 1, 0), (2, 300, 3, 2, 4), (1, 130, 2, 3, 4)])
def test_whole_layer_calls_give_the_bits_of_the_separate_steps(batch, seq, layers, heads, experts):
    """One native call per layer and direction against one autograd node per step: the same kernels on the same operands (the weight
    gradients of layers as small as these leave in one grouped launch), so losses agree bit for bit and matrix gradients up to the
    order in which split-K sums meet.  130 rows take the separate rotation kernel (products below the 2-CTA tiles), 993 end inside a
    tile, 903 x 3 leaves the row statistics at odd offsets."""
    _assert_whole_layers_match_the_steps(_layers_cfg(heads, layers, 512 * heads, experts), batch, seq)


@pytest.mark.parametrize("group", [0.0, float("inf")])
@pytest.mark.parametrize("heads,mlp,experts", [(2, 1024, 0), (2, 1288, 0), (2, 520, 0), (1, 2048, 0), (2, 1024, 4)])
def test_whole_layer_calls_with_grouped_and_separate_weight_gradients(monkeypatch, group, heads, mlp, experts):
    """Both scratch layouts of the backward call, with MLPs of four widths, wider and narrower: d_h over d_qkv and the value rows, or in
    a place of its own."""
    from autoresearch_b200.ops import sm100
    monkeypatch.setattr(sm100, "GROUP_DW_FLOPS", group)
    _assert_whole_layers_match_the_steps(_layers_cfg(heads, 3, mlp, experts), 3, 331)


def test_captured_pass_follows_its_inputs():
    """A training pass (forward, backward into main gradients) captured in a CUDA graph, with its early-started kernels, and
    replayed on other tokens, against the same pass run directly: losses bit for bit, gradients up to the order of split-K sums."""
    from autoresearch_b200.config import model_preset
    from autoresearch_b200.ops import kernels as K
    cfg = model_preset("small")
    torch.manual_seed(5)
    mod = _build("sm100", cfg, torch.bfloat16)
    for p in mod.parameters():
        p.main_grad = torch.zeros(p.shape, dtype=torch.float32, device="cuda")
    batches = [torch.randint(0, cfg.vocab, (2, 2, 200), device="cuda", dtype=torch.int32) for _ in range(3)]
    ids, tgt = batches[0][0].clone(), batches[0][1].clone()

    def step():
        for p in mod.parameters():
            p.main_grad.zero_()
        loss, per_tok = mod(ids, tgt, grad_scale=1.0 / ids.numel())
        loss.backward()
        return per_tok

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step()
    for b in batches[1:]:
        ids.copy_(b[0]); tgt.copy_(b[1])
        graph.replay()
        got = out.clone(), [p.main_grad.clone() for p in mod.parameters()]
        want = step()
        assert torch.equal(got[0], want)
        for p, g in zip(mod.parameters(), got[1]):
            assert (p.main_grad - g).norm() <= 1e-3 * p.main_grad.norm() + 1e-9
    K.check_err_flag()


class _TrainingPass:
    """A small model with value embeddings in half of its layers and fp32 main gradients; ``run`` is one forward and backward pass
    on the staged ids."""

    def __init__(self, seed=5):
        from autoresearch_b200.config import model_preset
        self.cfg = model_preset("small")
        torch.manual_seed(seed)
        self.mod = _build("sm100", self.cfg, torch.bfloat16)
        for p in self.mod.parameters():
            p.main_grad = torch.zeros(p.shape, dtype=torch.float32, device="cuda")
        self.ids, self.tgt = self.batch(), self.batch()

    def batch(self):
        return torch.randint(0, self.cfg.vocab, (2, 200), device="cuda", dtype=torch.int32)

    def run(self):
        for p in self.mod.parameters():
            p.main_grad.zero_()
        loss, _ = self.mod(self.ids, self.tgt, grad_scale=1.0 / self.ids.numel())
        loss.backward()

    def embedding_grads(self):
        names = {n: p.main_grad for n, p in self.mod.named_parameters() if n == "wte" or n.endswith(".ve")}
        assert len(names) > 1
        return {n: g.clone() for n, g in names.items()}


def _assert_same_embedding_grads(got, want):
    for n in want:      # their sums have a fixed order; what they sum differs by the order of split-K sums below
        assert (got[n] - want[n]).norm() <= 1e-3 * want[n].norm() + 1e-9, n


def test_direct_pass_on_the_capture_stream_does_not_take_the_captured_plan():
    """Capture on an explicit stream, then the same pass directly on that stream, ids untouched, before any replay: every captured
    or direct pass makes one plan of its own, shared by the word and the value embeddings."""
    from autoresearch_b200.ops import kernels as K
    t = _TrainingPass()
    side = torch.cuda.Stream()
    made, make = [], K._embedding_plan
    K._embedding_plan = lambda ids, vocab: made.append(torch.cuda.is_current_stream_capturing()) or make(ids, vocab)
    try:
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            t.run()
            want = t.embedding_grads()
            graph = torch.cuda.CUDAGraph()
            graph.capture_begin()
            t.run()
            graph.capture_end()
            t.run()
            got = t.embedding_grads()
            graph.replay()
            replayed = t.embedding_grads()
        side.synchronize()
    finally:
        K._embedding_plan = make
    assert made == [False, True, False]
    assert len(K._emb_plan) == 0
    _assert_same_embedding_grads(got, want)
    _assert_same_embedding_grads(replayed, want)
    K.check_err_flag()


def test_steps_of_one_pass_share_a_plan_and_a_block_called_by_itself_makes_its_own(monkeypatch):
    from autoresearch_b200.ops import kernels as K
    t = _TrainingPass()
    be, cfg = t.mod.backend, t.cfg
    be.layer_calls = False
    made, make = [], K._embedding_plan
    monkeypatch.setattr(K, "_embedding_plan", lambda ids, vocab: made.append(1) or make(ids, vocab))
    t.run()
    assert len(made) == 1
    blk = next(b for b in t.mod.blocks if b.ve is not None)
    B, T = t.ids.shape
    for n in (2, 3):
        xn = torch.randn(B * T, cfg.d_model, device="cuda").to(torch.bfloat16).requires_grad_()
        be.attention_block(xn, blk, t.ids.reshape(-1), B, T, cfg, t.mod.rope_cos, t.mod.rope_sin, T).float().sum().backward()
        assert len(made) == n and len(K._emb_plan) == 0
    K.check_err_flag()


def test_direct_pass_after_a_replay_that_refills_the_ids():
    """The captured pass copies its ids in, which raises no version at replay; a direct pass then sees the new ids."""
    from autoresearch_b200.ops import kernels as K
    t = _TrainingPass()
    source = t.ids.clone()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        t.run()
        graph = torch.cuda.CUDAGraph()
        graph.capture_begin()
        t.ids.copy_(source)
        t.run()
        graph.capture_end()
        graph.replay()
        t.run()
        source.copy_(t.batch())
        graph.replay()
        replayed = t.embedding_grads()
        t.run()
        got = t.embedding_grads()
        t.ids = t.ids.clone()
        t.run()
        want = t.embedding_grads()
    side.synchronize()
    _assert_same_embedding_grads(replayed, want)
    _assert_same_embedding_grads(got, want)
    K.check_err_flag()


def test_two_streams_with_one_set_of_ids():
    """Passes of two models on the same ids, queued on two streams without waiting for each other."""
    from autoresearch_b200.ops import kernels as K
    a, b = _TrainingPass(5), _TrainingPass(6)
    b.ids, b.tgt = a.ids, a.tgt
    want = []
    for t in (a, b):
        t.run()
        want.append(t.embedding_grads())
    streams = [torch.cuda.Stream() for _ in range(2)]
    for s in streams:
        s.wait_stream(torch.cuda.current_stream())
    for _ in range(3):
        for t, s in zip((a, b), streams):
            with torch.cuda.stream(s):
                t.run()
    torch.cuda.synchronize()
    for t, w in zip((a, b), want):
        _assert_same_embedding_grads(t.embedding_grads(), w)
    K.check_err_flag()


@pytest.mark.parametrize("heads,mlp,experts", [(2, 1024, 0), (3, 768, 0), (1, 1024, 0), (2, 1024, 4)])
def test_scoring_pass_holds_no_more_memory_than_the_separate_steps(heads, mlp, experts):
    """Peak of the layers of a pass without gradients, whole-layer calls against one call per step, and the same bits: MLPs of four,
    two and eight widths, and experts.  The row statistics lie over the MLP part unless that is narrow: 16 bytes a row and head."""
    from autoresearch_b200.config import ModelConfig, MoEConfig
    moe = MoEConfig(n_experts=experts, top_k=2, mlp_dim_e=mlp, capacity_factor=1.25) if experts else None
    cfg = ModelConfig(vocab=512, seq_len=2048, d_model=128 * heads, n_head=heads, head_dim=128, mlp_dim=mlp, n_layer=3, moe=moe)
    torch.manual_seed(7)
    mod = _build("sm100", cfg, torch.bfloat16)
    B, T = 8, 2048
    ids = torch.randint(0, cfg.vocab, (B, T), device="cuda", dtype=torch.int32)
    peak, out = {}, {}
    with torch.no_grad():
        x = mod.embed(ids)
        for whole in (True, False):
            mod.backend.layer_calls = whole
            for _ in range(2):                   # first pass: lazily made buffers
                torch.cuda.synchronize()
                torch.cuda.reset_peak_memory_stats()
                before = torch.cuda.memory_allocated()
                out[whole] = None
                out[whole] = mod.run_layers(x, x, ids, B, T)
                torch.cuda.synchronize()
                peak[whole] = torch.cuda.max_memory_allocated() - before
    assert torch.equal(out[True], out[False])
    assert peak[True] <= peak[False] + 16 * B * T * heads + (1 << 21), peak


@pytest.mark.parametrize("group", [0.0, 6e10])
def test_training_pass_keeps_no_more_per_layer_than_the_separate_steps(monkeypatch, group):
    """Peak of forward and backward through six layers: what a layer keeps may not exceed what the separate steps keep (a width of D
    more in each would be six).  Beside it the call in progress holds its scratch, M + 5 D columns (ungrouped max(M, 4 D) + D), the gate's
    32, the statistics and two input gradients, where the separate steps' widest moment is d_h and its product, 5 D: with M = 4 D and
    D = 256 that is 6 widths (2) and less than a quarter."""
    from autoresearch_b200.config import ModelConfig
    from autoresearch_b200.ops import sm100
    monkeypatch.setattr(sm100, "GROUP_DW_FLOPS", group)
    heads, B, T = 2, 8, 2048
    D = 128 * heads
    cfg = ModelConfig(vocab=512, seq_len=T, d_model=D, n_head=heads, head_dim=128, mlp_dim=4 * D, n_layer=6)
    mod = _build("sm100", cfg, torch.bfloat16)
    for p in mod.parameters():
        p.main_grad = torch.zeros(p.shape, dtype=torch.float32, device="cuda")
    ids = torch.randint(0, cfg.vocab, (B, T), device="cuda", dtype=torch.int32)
    x = torch.randn(B * T, D, device="cuda").to(torch.bfloat16).requires_grad_()
    g = torch.randn(B * T, D, device="cuda").to(torch.bfloat16)
    kept, peak = {}, {}
    for whole in (True, False):
        mod.backend.layer_calls = whole
        for _ in range(2):
            x.grad = None
            torch.cuda.reset_peak_memory_stats()
            before = torch.cuda.memory_allocated()
            out = mod.run_layers(x, x, ids, B, T)
            kept[whole] = torch.cuda.memory_allocated() - before
            out.backward(g)
            del out
            torch.cuda.synchronize()
            peak[whole] = torch.cuda.max_memory_allocated() - before
    width = B * T * D * 2
    assert kept[True] <= kept[False] + width // 4, (kept, width)
    assert peak[True] <= peak[False] + (6 if group else 2) * width + width // 4 + (1 << 21), (peak, width)

"""Which small groups the one-launch Muon step takes: its kernel reads fp32 state through pointers, and what the tensor operations
accepted beside that still goes to them."""
import pytest
import torch

from autoresearch_b200.ops import kernels as K, sm100
from autoresearch_b200.optim import muon_adamw as MA


class _Library:
    def __init__(self):
        self.calls = 0

    def arb_muon_small(self, *args):
        self.calls += 1
        return 0 if args[5] > 0 else -3          # the number of matrices


def _group(G, m, n, **dtypes):
    g = torch.Generator().manual_seed(G + m + n)
    st = dict(master=torch.randn(G, m, n, generator=g), momentum=torch.randn(G, m, n, generator=g) * 0.01,
              second=torch.rand((G, m, 1) if m >= n else (G, 1, n), generator=g))
    st = {k: v.to(dtypes.get(k, torch.float32)) for k, v in st.items()}
    return st, torch.randn(G, m, n, generator=g) * 0.01, st["master"].to(torch.bfloat16)


@pytest.mark.parametrize("G,dtypes,native", [(3, {}, True), (0, {}, False), (3, dict(momentum=torch.bfloat16), False),
                                             (3, dict(second=torch.float64), False), (3, dict(master=torch.float64), False)])
def test_one_launch_takes_fp32_state_only(monkeypatch, G, dtypes, native):
    fake = _Library()
    monkeypatch.setattr(K, "lib", lambda: fake)
    monkeypatch.setattr(K, "_stream", lambda: 0)
    st, grad, pv = _group(G, 4, 32, **dtypes)
    want = {k: v.clone() for k, v in st.items()}
    sm100.OptimKernels().muon_group(st, grad, pv, 0.9, 0.02, 0.1, 0.95, 5)
    assert fake.calls == int(native)
    if native:
        return
    u = MA.muon_nesterov(want["momentum"], grad, 0.9, torch.bfloat16)
    MA.cautious_update(want["master"], MA.normuon(MA.newton_schulz(MA.frob_normalise(u), 5), want["second"], 0.95), 0.02, 0.1)
    for k in want:
        assert torch.equal(st[k], want[k]), k
    assert torch.equal(pv, st["master"].to(torch.bfloat16))

"""Into what memory the native layer call adds its weight gradients.  A stand-in for the call adds one to every element of the buffers
it is given, on the CPU; the GEMM of the separate steps takes fp32 gradients of the parameter's shape, rows at any stride, and refuses
others."""
import ctypes as C
from types import SimpleNamespace

import pytest
import torch

from autoresearch_b200.ops import kernels as K, sm100

PARAMS = ("lam_r", "lam_0", "wqkv", "wo", "wfc", "wdn")


@pytest.fixture
def call(monkeypatch):
    """backward(main gradients by name) of a layer of width 128: the parameters, after the stand-in has run."""
    N, D, M = 4, 128, 512
    shapes = dict(lam_r=(3,), lam_0=(3,), wqkv=(3 * D, D), wo=(D, D), wfc=(M, D), wdn=(D, M))

    def layer_call(entry, pointers, sizes, eps, scale):
        for ptr, name in zip(pointers[-7:-1], PARAMS):
            n = int(torch.Size(shapes[name]).numel())
            buf = (C.c_float * n).from_address(ptr)
            for i in range(n):
                buf[i] += 1.0

    monkeypatch.setattr(K, "layer_call", layer_call)
    monkeypatch.setattr(K, "err_flag", lambda device=None: torch.zeros(1, dtype=torch.int32))

    def backward(mains):
        ps = {n: torch.zeros(s, dtype=torch.bfloat16) for n, s in shapes.items()}
        for n, m in mains.items():
            ps[n].main_grad = m
        x, aux = torch.zeros(N, D, dtype=torch.bfloat16), torch.zeros(64, dtype=torch.bfloat16)
        ctx = SimpleNamespace(saved_tensors=(x, x, *ps.values(), None, None, None, aux, aux, aux, None), eps=1e-5,
                              sizes=(1, N, 1, M, N, 0, 32, 0, 1, 0, 0), chain=SimpleNamespace(buf=None))
        return dict(zip(PARAMS, sm100._layer_backward(ctx, x, None)[2]))
    return backward


def test_strided_main_gradients_take_the_sum_and_nothing_beside_them_changes(call):
    wide = torch.zeros(384, 160)
    dense = torch.zeros(128, 128)
    grads = call(dict(wqkv=wide[:, :128], wo=dense))
    assert (wide[:, :128] == 1).all() and (wide[:, 128:] == 0).all()
    assert (dense == 1).all()
    assert grads["wqkv"] is None and grads["wo"] is None
    assert (grads["wfc"] == 1).all() and grads["wfc"].dtype is torch.bfloat16


@pytest.mark.parametrize("main", [torch.zeros(128, 128, dtype=torch.bfloat16), torch.zeros(128, 64), torch.zeros(128 * 128),
                                  torch.zeros(128, 128, device="meta")])
def test_main_gradients_that_the_products_cannot_add_into_are_refused(call, main):
    with pytest.raises(ValueError):
        call(dict(wo=main))


@pytest.mark.parametrize("mode,grouped", [(0, True), (1, False), (2, True)])
def test_grouped_weight_gradients_follow_the_tile_mode(monkeypatch, mode, grouped):
    """The grouped launch has 2-CTA tiles: with the mode that asks for 1-CTA tiles the gradients stay separate products."""
    seen = []
    monkeypatch.setattr(K, "layer_call", lambda entry, pointers, sizes, eps, scale: seen.append(sizes))
    monkeypatch.setattr(K, "err_flag", lambda device=None: torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(K, "_gemm_mode", mode)
    D, M = 128, 512
    w = lambda *s: torch.zeros(*s, dtype=torch.bfloat16)
    ctx = SimpleNamespace(save_for_backward=lambda *t: None)
    sm100._layer_forward(ctx, w(4, D), w(4, D), w(1), w(1), w(3 * D, D), w(D, D), w(M, D), w(D, M), None, None, w(4), w(4, 64), w(4, 64),
                         1, 4, 4, 0, 32, 1e-5, None, False, None)
    assert [s[8] for s in seen] == [int(grouped)]

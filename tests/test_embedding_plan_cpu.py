"""Whose tables an embedding gradient is summed by: a stand-in for the native library records which plan every call is given, so
neither a GPU nor the built library is needed."""
import ctypes as C

import pytest
import torch

from autoresearch_b200.ops import kernels as K


class _Library:
    """Counts plans and remembers the sort order handed to each gradient; `capture` is the capture id of the stream (0: none)."""

    def __init__(self):
        self.plans, self.used, self.capture = [], [], 0

    def arb_capture_id(self, out, stream):
        C.cast(out, C.POINTER(C.c_ulonglong))[0] = self.capture
        return 0

    def arb_embedding_plan(self, ids, n, vocab, rows, n_max, hist, perm, *tables):
        self.plans.append((self.capture, perm))
        return 0

    def arb_embedding_bwd_sorted(self, perm, *rest):
        self.used.append(perm)
        return 0


class _Pass:
    """Stands for what the nodes of one forward pass share."""


@pytest.fixture
def lib(monkeypatch):
    fake = _Library()
    monkeypatch.setattr(K, "lib", lambda: fake)
    monkeypatch.setattr(K, "_stream", lambda: 7)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: fake.capture != 0)
    K._emb_plan.clear()
    yield fake
    K._emb_plan.clear()


def _args(n=40, vocab=8, d=16):
    return torch.arange(n, dtype=torch.int32) % vocab, torch.zeros(n, d, dtype=torch.bfloat16), torch.zeros(vocab, d)


def test_a_plan_recorded_under_capture_serves_no_call_outside(lib):
    """The kernels of a captured plan run at replay: until then its tables are uninitialised memory."""
    ids, g, dw = _args()
    lib.capture = 3
    K.embedding_bwd(ids, g, dw)
    lib.capture = 0
    K.embedding_bwd(ids, g, dw)
    assert [c for c, _ in lib.plans] == [3, 0]
    assert lib.used == [p for _, p in lib.plans]


def test_a_later_pass_on_the_same_ids_makes_its_own_plan(lib):
    """A graph replay or a raw-pointer writer refills ids without raising their version: what an earlier pass found is not asked."""
    ids, g, dw = _args()
    for _ in range(3):
        K.embedding_bwd(ids, g, dw)
    assert len(lib.plans) == 3


def test_gradients_of_one_pass_share_a_plan_per_capture_and_it_goes_with_the_pass(lib):
    ids, g, dw = _args()
    one, other = _Pass(), _Pass()
    for _ in range(3):
        K.embedding_bwd(ids, g, dw, one)
    assert len(lib.plans) == 1
    K.embedding_bwd(ids, g, dw, other)                       # the next forward pass, while the graph of the first is alive
    assert len(lib.plans) == 2
    for lib.capture in (5, 6):                               # two captures of one retained graph
        K.embedding_bwd(ids, g, dw, one)
        K.embedding_bwd(ids, g, dw, one)
    assert [c for c, _ in lib.plans] == [0, 0, 5, 6]
    lib.capture = 0
    ids.add_(0)                                              # refilled in place
    K.embedding_bwd(ids, g, dw, one)
    K.embedding_bwd(ids, g, torch.zeros(9, 16), one)         # another vocabulary
    assert len(lib.plans) == 6
    del one, other
    assert len(K._emb_plan) == 0


def test_ids_without_a_version_counter(lib):
    ids, g, dw = _args()
    with torch.inference_mode():
        fixed = ids + 0
    p = _Pass()
    K.embedding_bwd(fixed, g, dw, p)
    K.embedding_bwd(fixed, g, dw, p)
    assert len(lib.plans) == 1


def test_plans_are_dropped_when_their_last_gradient_has_been_launched(lib):
    ids, g, dw = _args()
    p = _Pass()
    K.embedding_bwd(ids, g, dw, p)
    K.forget_embedding_plans(p)
    K.forget_embedding_plans(p)
    K.forget_embedding_plans(None)
    assert len(K._emb_plan) == 0

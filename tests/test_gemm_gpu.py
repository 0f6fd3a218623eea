"""tcgen05 GEMM against a plain fp32 PyTorch matmul of the same bf16 operands."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True, params=[1, 2, 0], ids=["one_cta", "cta_pair", "auto"])
def tile_mode(request):
    """Every case runs on the 1-CTA kernel, on the 2-CTA (cta_group::2) kernel and with the
    automatic choice."""
    from autoresearch_b200.ops import kernels as K_
    K_.gemm_set_mode(request.param)
    yield request.param
    K_.gemm_set_mode(0)


def _rand(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).to(torch.bfloat16)


def _close(out, ref, tol=2e-2):
    err = (out.float() - ref).abs().max().item()
    den = ref.abs().max().item() + 1e-6
    assert err / den < tol, f"rel err {err / den:.4g}"


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 512, 256), (384, 128, 192), (200, 328, 136),
                                   (1024, 1024, 1024), (129, 72, 520)])
def test_nt(M, N, K):
    from autoresearch_b200.ops import kernels as K_
    torch.manual_seed(0)
    a, b = _rand(M, K), _rand(N, K)
    out = K_.gemm(a, b)
    _close(out, a.float() @ b.float().t())
    K_.check_err_flag()


@pytest.mark.parametrize("M,N,K", [(256, 256, 128), (200, 328, 136), (512, 1024, 768)])
def test_nn(M, N, K):
    from autoresearch_b200.ops import kernels as K_
    torch.manual_seed(1)
    a, b = _rand(M, K), _rand(K, N)
    out = K_.gemm(a, b, trans_b=False)
    _close(out, a.float() @ b.float())


@pytest.mark.parametrize("M,N,K", [(256, 256, 128), (264, 136, 1000), (1024, 512, 4096)])
def test_tn_atomic_accumulate(M, N, K):
    from autoresearch_b200.ops import kernels as K_
    torch.manual_seed(2)
    a, b = _rand(K, M), _rand(K, N)
    acc = torch.randn(M, N, device="cuda")
    ref = acc.clone() + a.float().t() @ b.float()
    K_.gemm(a, b, trans_a=True, trans_b=False, out=acc, epi=K_.EPI_ATOMIC_F32)
    _close(acc, ref, 1e-2)
    # explicit split-K
    acc2 = torch.zeros(M, N, device="cuda")
    K_.gemm(a, b, trans_a=True, trans_b=False, out=acc2, epi=K_.EPI_ATOMIC_F32, splitk=3)
    _close(acc2, a.float().t() @ b.float(), 1e-2)


def test_tn_nt_mixed_and_f32_store():
    from autoresearch_b200.ops import kernels as K_
    torch.manual_seed(3)
    a, b = _rand(320, 192), _rand(256, 320)      # A = a^T [192, 320], B = b^T
    out = K_.gemm(a, b, trans_a=True, trans_b=True, epi=K_.EPI_STORE_F32)
    _close(out, a.float().t() @ b.float().t(), 1e-2)


def test_epilogues():
    from autoresearch_b200.ops import kernels as K_
    torch.manual_seed(4)
    M, N, Kd = 256, 384, 128
    a, b = _rand(M, Kd, scale=0.3), _rand(N, Kd, scale=0.3)
    ref = a.float() @ b.float().t()
    _close(K_.gemm(a, b, epi=K_.EPI_RELU2), torch.relu(ref) ** 2)
    aux = _rand(M, N)
    _close(K_.gemm(a, b, epi=K_.EPI_ADD_AUX, aux=aux), ref + aux.float())
    act = (torch.relu(aux.float()) ** 2).to(torch.bfloat16)
    _close(K_.gemm(a, b, epi=K_.EPI_RELU2_BWD, aux=act), ref * 2 * torch.sqrt(act.float()))
    sq = _rand(256, 256, scale=0.1)
    got = K_.gemm(sq, sq, epi=K_.EPI_NS_COMBINE, aux=sq, alpha=1.5, beta=-2.0, gamma=0.5)
    want = 1.5 * torch.eye(256, device="cuda") - 2.0 * sq.float() + 0.5 * (sq.float() @ sq.float().t())
    _close(got, want)


def test_batched():
    from autoresearch_b200.ops import kernels as K_
    torch.manual_seed(5)
    G, m, n = 5, 256, 512
    x = _rand(G, m, n, scale=0.2)
    A = K_.gemm(x, x)                                        # X X^T
    _close(A, x.float() @ x.float().transpose(1, 2))
    At = K_.gemm(x, x, trans_a=True, trans_b=False)          # X^T X
    _close(At, x.float().transpose(1, 2) @ x.float())
    y = K_.gemm(A, x, trans_b=False)                         # A X
    _close(y, A.float() @ x.float())


def test_strided_views():
    """Operands that are column blocks of a wider buffer (packed qkv) and row slices."""
    from autoresearch_b200.ops import kernels as K_
    torch.manual_seed(6)
    big = _rand(512, 768)
    w = _rand(256, 256)
    a = big[:, 256:512]
    _close(K_.gemm(a, w), a.float() @ w.float().t())
    out = torch.zeros(512, 512, dtype=torch.bfloat16, device="cuda")
    K_.gemm(a, w, out=out[:, 256:])
    _close(out[:, 256:], a.float() @ w.float().t())
    assert out[:, :256].abs().max().item() == 0


def test_rejects_bad_arguments():
    from autoresearch_b200.ops import kernels as K_
    a, b = _rand(128, 60), _rand(128, 60)      # K not a multiple of 8
    with pytest.raises(K_.KernelError):
        K_.gemm(a, b)


@pytest.mark.parametrize("shape", [(1024, 512, 256), (192, 128, 64), (4096, 3072, 1024)])
def test_gemm_pulls_its_b_operand_in_the_prologue(shape):
    """A registered pending pull makes the GEMM copy its B operand from another buffer first (the mechanism
    that fuses the parameter all-gather into the first consuming GEMM); here the source is local memory."""
    from autoresearch_b200.ops import kernels as K
    M, N, Kd = shape
    torch.manual_seed(3)
    x = torch.randn(M, Kd, device="cuda").to(torch.bfloat16)
    w_new = (torch.randn(N, Kd, device="cuda") * 0.05).to(torch.bfloat16)
    w = torch.zeros_like(w_new)                       # stale local copy
    K.pending_pulls[w.data_ptr()] = (w_new.data_ptr(), w.numel() * 2)
    for _ in range(3):                                # the counter barrier must work launch after launch
        y = K.gemm(x, w)
        torch.cuda.synchronize()
        K.check_err_flag()
        assert w.data_ptr() not in K.pending_pulls
        assert torch.equal(w, w_new)
        ref = x.float() @ w_new.float().t()
        assert ((y.float() - ref).norm() / ref.norm()).item() < 1e-2
        w.zero_()
        K.pending_pulls[w.data_ptr()] = (w_new.data_ptr(), w.numel() * 2)
    K.flush_pending_pulls()
    torch.cuda.synchronize()
    assert torch.equal(w, w_new) and not K.pending_pulls


@pytest.mark.parametrize("shape", [(1024, 512, 256), (4096, 3072, 1024)])
def test_gemm_copies_the_next_operand_while_it_computes(shape):
    """With two operands pending, the first GEMM copies its own B in the prologue and, in a spare warp, the
    OTHER pending operand while its tiles run; the second GEMM then finds its operand local already."""
    from autoresearch_b200.ops import kernels as K
    M, N, Kd = shape
    torch.manual_seed(4)
    x = torch.randn(M, Kd, device="cuda").to(torch.bfloat16)
    new = [(torch.randn(N, Kd, device="cuda") * 0.05).to(torch.bfloat16) for _ in range(2)]
    # the second operand's size is not a multiple of the copy loop's stride: exercises its tail
    new.append((torch.randn(N + 8, Kd, device="cuda") * 0.05).to(torch.bfloat16))
    stale = [torch.zeros_like(w) for w in new]
    K.pending_pulls.clear()
    for s, w in zip(stale, new):
        K.pending_pulls[s.data_ptr()] = (w.data_ptr(), w.numel() * 2)
    K.pull_stream = K._stream()
    y0 = K.gemm(x, stale[0])
    assert len(K.pending_pulls) == 1                  # own operand + one ahead
    torch.cuda.synchronize()
    assert torch.equal(stale[0], new[0]) and torch.equal(stale[1], new[1]) and stale[2].abs().max().item() == 0
    y1 = K.gemm(x, stale[1])                          # nothing pending for it; copies operand 2 ahead
    assert not K.pending_pulls
    y2 = K.gemm(x, stale[2])
    torch.cuda.synchronize()
    K.check_err_flag()
    assert torch.equal(stale[2], new[2])
    for y, w in zip((y0, y1, y2), new):
        ref = x.float() @ w.float().t()
        assert ((y.float() - ref).norm() / ref.norm()).item() < 1e-2
    # a GEMM on another stream leaves the ahead copies to the stream they were registered on
    stale[1].zero_()
    K.pending_pulls[stale[1].data_ptr()] = (new[1].data_ptr(), new[1].numel() * 2)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        K.gemm(x, stale[0])
    assert len(K.pending_pulls) == 1
    K.flush_pending_pulls()
    torch.cuda.synchronize()
    assert torch.equal(stale[1], new[1])


@pytest.mark.parametrize("mode", [1, 2])
def test_ragged_batches_skip_rows_beyond_the_valid_count(mode):
    """Grouped expert GEMM: per-item row counts (device array), several row slabs per weight matrix; tiles beyond the
    count are left untouched and the K range of the transposed product is cut to the valid rows."""
    from autoresearch_b200.ops import kernels as K
    torch.manual_seed(7)
    E, W, cap, D, M = 2, 3, 640, 256, 512          # E weights, W slabs each, cap rows per slab
    G = E * W
    counts = torch.tensor([640, 0, 130, 257, 512, 5], dtype=torch.int32, device="cuda")
    x = (torch.randn(G, cap, D, device="cuda") * 0.5).to(torch.bfloat16)
    for g in range(G):                               # rows between the count and the next tile boundary are zero
        x[g, int(counts[g]):] = 0
    w = (torch.randn(E, M, D, device="cuda") * 0.1).to(torch.bfloat16)
    K.gemm_set_mode(mode)
    try:
        out = torch.full((G, cap, M), 7.0, dtype=torch.bfloat16, device="cuda")
        K.gemm(x, w, out=out, epi=K.EPI_RELU2, m_valid=counts, b_div=W)
        tile = 256 if mode == 2 else 128
        for g in range(G):
            c = int(counts[g])
            ref = torch.relu(x[g, :c].float() @ w[g // W].float().t()) ** 2
            if c:
                assert ((out[g, :c].float() - ref).norm() / ref.norm()).item() < 1e-2
            done = (c + tile - 1) // tile * tile
            assert (out[g, min(done, cap):] == 7.0).all()           # untouched
            assert (out[g, c:min(done, cap)] == 0).all()            # computed from zero rows
        # dW[e] += sum over the slabs of e of dy^T x, K cut to the valid rows; poison what lies beyond the padding
        dy = (torch.randn(G, cap, M, device="cuda") * 0.1).to(torch.bfloat16)
        for g in range(G):
            c = int(counts[g])
            dy[g, c:] = 0
            pad = (c + 63) // 64 * 64
            dy[g, pad:] = float("nan")
            x[g, pad:] = float("nan")
        dw = torch.zeros(E, M, D, dtype=torch.float32, device="cuda")
        K.gemm(dy.view(E, W * cap, M), x.view(E, W * cap, D), trans_a=True, trans_b=False, out=dw, epi=K.EPI_ATOMIC_F32,
               k_valid=counts.view(E, W).contiguous(), k_seg=cap)
        torch.cuda.synchronize()
        K.check_err_flag()
        for e in range(E):
            ref = sum(dy[e * W + j, :int(counts[e * W + j])].float().t() @ x[e * W + j, :int(counts[e * W + j])].float()
                      for j in range(W))
            assert torch.isfinite(dw[e]).all()
            assert ((dw[e] - ref).norm() / ref.norm()).item() < 1e-2
    finally:
        K.gemm_set_mode(0)


@pytest.mark.parametrize("G,d,k", [(1, 512, 512), (3, 520, 264), (2, 776, 1024), (5, 1024, 128), (1, 2048, 256), (2, 256, 512), (1, 1288, 72)])
def test_symmetric_products_mirror_their_upper_tiles(G, d, k):
    """Gram matrices in both layouts and the Newton-Schulz combination, against the same products with every tile computed: each
    element is the same sum in the same order, so the bits are equal (sizes with one tile, ragged last tiles, many tiles)."""
    from autoresearch_b200.ops import kernels as K
    torch.manual_seed(d + k)
    x = (torch.randn(G, d, k, device="cuda") * 0.1).to(torch.bfloat16)
    xt = x.transpose(1, 2).contiguous()
    for a, kw in ((x, {}), (xt, dict(trans_a=True, trans_b=False))):
        full = K.gemm(a, a, **kw)
        buf = torch.full((G, d + 2, d), 3.0, device="cuda", dtype=torch.bfloat16)
        half = buf[:, 1:-1]
        K.gemm(a, a, out=half, epi=K.EPI_SYM_STORE, **kw)
        assert torch.equal(full, full.transpose(1, 2)) and torch.equal(half, full)
        assert (buf[:, 0] == 3.0).all() and (buf[:, -1] == 3.0).all()
    args = dict(aux=full, alpha=3.4, beta=-4.7, gamma=2.0)
    assert torch.equal(K.gemm(full, full, epi=K.EPI_NS_COMBINE, **args), K.gemm(full, full, epi=K.EPI_SYM_NS_COMBINE, **args))
    K.check_err_flag()


@pytest.mark.parametrize("M,N,Kd", [(512, 256, 64), (2048, 512, 1536), (1544, 1416, 200), (512, 4736, 128), (640, 3840, 72)])
def test_few_tiles_and_just_too_many(M, N, Kd):
    """Products around the 148 tiles of 128 x 128 where the tile choice changes (148 and 150 tiles in the last two), with every
    bf16 epilogue that both kernels have: bf16 outputs of K products, 1e-2."""
    from autoresearch_b200.ops import kernels as K
    torch.manual_seed(M + N)
    a, w = torch.randn(M, Kd, device="cuda").bfloat16(), (torch.randn(N, Kd, device="cuda") / Kd ** 0.5).bfloat16()
    x = torch.rand(M, N, device="cuda").bfloat16()
    acc = a.float() @ w.float().t()
    for epi, ref in ((K.EPI_STORE_BF16, acc), (K.EPI_RELU2, acc.clamp_min(0) ** 2), (K.EPI_ADD_AUX, acc + x.float()),
                     (K.EPI_RELU2_BWD, acc * 2 * x.float().sqrt())):
        out = K.gemm(a, w, epi=epi, aux=x if epi in (K.EPI_ADD_AUX, K.EPI_RELU2_BWD) else None)
        assert ((out.float() - ref).norm() / ref.norm()).item() < 1e-2
    out = K.gemm(a, w.t().contiguous(), trans_b=False)
    assert ((out.float() - acc).norm() / acc.norm()).item() < 1e-2
    K.check_err_flag()


@pytest.mark.parametrize("own_stream", [False, True])
@pytest.mark.parametrize("Kd,shapes", [(1, [(8, 8)]), (130, [(256, 256), (264, 512)]), (2048, [(1536, 512), (2048, 512), (512, 2048), (512, 512)]),
                                       (993, [(1152, 384), (1536, 384), (384, 1536), (384, 384)]), (8000, [(128, 128), (384, 128), (512, 128)])])
def test_grouped_weight_gradients(Kd, shapes, own_stream):
    """One launch against 64 bits: one row, ragged tiles and K, splits that do and do not divide the K blocks; fp32 sums of Kd
    products of bf16 values, and rows around the outputs that stay untouched; on the default stream and on another, whose operands are
    made on it just before."""
    import ctypes as C
    from contextlib import nullcontext
    with torch.cuda.stream(torch.cuda.Stream()) if own_stream else nullcontext():
        _grouped_weight_gradients(C, Kd, shapes)


def _grouped_weight_gradients(C, Kd, shapes):
    from autoresearch_b200.ops import kernels as K
    torch.manual_seed(Kd)
    dy = [torch.randn(Kd, m, device="cuda").bfloat16() for m, _ in shapes]
    x = [torch.randn(Kd, n, device="cuda").bfloat16() for _, n in shapes]
    buf = [torch.full((m + 2, n), 0.25, device="cuda") for m, n in shapes]
    out = [b[1:-1] for b in buf]
    n = len(shapes)
    vec = lambda ts: (C.c_void_p * n)(*[t.data_ptr() for t in ts])
    ints = lambda v: (C.c_int * n)(*v)
    K._check(K.lib().arb_gemm_dw_group(vec(dy), vec(x), vec(out), ints([m for m, _ in shapes]), ints([c for _, c in shapes]), n, Kd,
                                       K.err_flag().data_ptr(), K._stream()), "gemm_dw_group")
    torch.cuda.synchronize()
    K.check_err_flag()
    for a, b, c, full in zip(dy, x, out, buf):
        ref = 0.25 + a.double().t() @ b.double()
        assert (c.double() - ref).abs().max() <= 2e-6 * (a.double().abs().t() @ b.double().abs()).max() + 1e-6
        assert (full[0] == 0.25).all() and (full[-1] == 0.25).all()


def test_symmetric_product_of_an_odd_side_writes_what_the_plain_product_writes():
    """The transposes are stored as pairs of rows: with an odd side the last pair would reach into the padding of a row.  Every tile is
    computed then, and the bits are those of the plain product, in the padding (whose rest of 16 bytes a tile store fills) too."""
    from autoresearch_b200.ops import kernels as K
    torch.manual_seed(11)
    d, ld = 1001, 1008
    x = (torch.randn(d, 128, device="cuda") * 0.1).to(torch.bfloat16)
    buf, aux, full = (torch.full((d, ld), 3.0, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    K.gemm(x, x, out=full[:, :d])
    K.gemm(x, x, out=buf[:, :d], epi=K.EPI_SYM_STORE)
    assert torch.equal(buf, full)
    aux[:, :d] = full[:, :d]
    got = []
    for epi in (K.EPI_NS_COMBINE, K.EPI_SYM_NS_COMBINE):
        got.append(torch.full_like(buf, 3.0))
        K.gemm(full[:, :d], full[:, :d], out=got[-1][:, :d], epi=epi, aux=aux[:, :d], alpha=3.4, beta=-4.7, gamma=2.0)
    assert torch.equal(*got)
    K.check_err_flag()

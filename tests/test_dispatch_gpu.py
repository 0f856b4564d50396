"""The rules that send a call to one kernel or another: sizes at the edges of each rule, against fp32 / fp64 PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ops():
    from oslo_b200 import ops
    from oslo_b200.ops import cuda_ops
    return ops, cuda_ops


def _rel(got, want):
    return float((got.double() - want.double()).norm() / want.double().norm())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("vocab,rows,with_bias", [(5, 40, True), (33, 130, False), (1003, 300, True), (1007, 257, False), (50257, 200, False)])
def test_loss_of_a_vocabulary_of_any_size(vocab, rows, with_bias, dtype):
    """Vocabulary sizes that are no multiple of 8: loss and gradients on the GEMM kernels, whose gradient matrix has padded rows.
    Each gradient is a sum of products of 16-bit factors rounded once more to 16 bits, so its 2-norm error is a few units of
    2^-9 (bf16) or 2^-12 (fp16); four units allowed."""
    ops, _ = _ops()
    gen = torch.Generator(device="cuda").manual_seed(vocab)
    mk = lambda *s, std: torch.randn(*s, device="cuda", generator=gen).mul_(std).to(dtype).requires_grad_(True)      # noqa: E731
    h, w = mk(rows, 256, std=0.5), mk(vocab, 256, std=0.1)
    b = mk(vocab, std=0.1) if with_bias else None
    lab = torch.randint(0, vocab, (rows,), device="cuda", generator=gen)
    lab[3], lab[4], lab[5] = -100, vocab - 1, 0
    before = ops.load_ext().launch_count()
    loss = ops.linear_cross_entropy(h, w, b, lab, chunk_rows=128)
    assert ops.load_ext().launch_count() > before
    (loss * 64).backward()
    leaves = [t.detach().double().requires_grad_(True) for t in ((h, w, b) if with_bias else (h, w))]
    logits = leaves[0] @ leaves[1].t() + (leaves[2] if with_bias else 0.0)
    want = torch.nn.functional.cross_entropy(logits, lab, ignore_index=-100)
    (want * 64).backward()
    unit = 2.0 ** (-9 if dtype == torch.bfloat16 else -12)
    assert abs(loss.item() - want.item()) < 16 * unit
    for got, leaf in zip((h, w, b), leaves):
        assert _rel(got.grad, leaf.grad) < 4 * unit, (vocab, got.shape, _rel(got.grad, leaf.grad))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("vocab, held", [(1003, False), (1007, True)])
def test_loss_gradient_sums_its_chunks_in_32_bits(vocab, held, dtype):
    """Sixteen row chunks into a gradient that lives in a flat buffer. One rounding to 16 bits has an rms error of 0.42 u of the value's
    (u = 2^-8 or 2^-11, mantissas of all kinds); the gradient matrix and the sum have one each, 0.6 u together, and an addition to a
    gradient of the same size one more at half the weight. 0.8 u allowed; sixteen roundings of growing sums come to 1.2 u and more."""
    ops, _ = _ops()
    gen = torch.Generator(device="cuda").manual_seed(vocab)
    mk = lambda *s, std: torch.randn(*s, device="cuda", generator=gen).mul_(std).to(dtype)      # noqa: E731
    h, w = mk(512, 256, std=0.5), mk(vocab, 256, std=0.1).requires_grad_(True)
    lab = torch.randint(0, vocab, (512,), device="cuda", generator=gen)
    wide = w.detach().double().requires_grad_(True)
    want, = torch.autograd.grad(torch.nn.functional.cross_entropy(h.double() @ wide.t(), lab) * 256, wide)
    base = torch.zeros_like(w) if not held else want.to(dtype)
    w.grad, w._oslo_accum_grad = base.detach().clone(), True
    (ops.linear_cross_entropy(h, w, None, lab, chunk_rows=32) * 256).backward()
    u = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    want = want + base.double()
    assert _rel(w.grad, want) < 0.8 * u, _rel(w.grad, want) / u


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("cols", [8, 256, 264, 512, 520, 768, 1024, 1032, 2048, 2056, 4096, 4104, 6144, 6152, 8192])
@pytest.mark.parametrize("rows", [1, 7, 1300])
def test_layernorm_rows_at_the_edges_of_its_layouts(rows, cols, dtype):
    """One size on each side of every (vectors per lane, warps per row) layout. Forward and input gradient are rounded once to the
    storage type; the weight gradients sum `rows` products in fp32 before that."""
    _, co = _ops()
    if dtype == torch.float32 and cols > 4096:
        pytest.skip("wider than the kernel takes in 32 bits")
    gen = torch.Generator(device="cuda").manual_seed(rows * 10007 + cols)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=gen)                                               # noqa: E731
    x, w, b, g = (mk(rows, cols) * 2 + 0.5).to(dtype), (1 + 0.1 * mk(cols)).to(dtype), mk(cols).to(dtype), mk(rows, cols).to(dtype)
    leaves = [t.clone().requires_grad_(True) for t in (x, w, b)]
    y = co.layer_norm(*leaves, 1e-5)
    y.backward(g)
    wide = [t.double().requires_grad_(True) for t in (x, w, b)]
    want = torch.nn.functional.layer_norm(wide[0], (cols,), wide[1], wide[2], 1e-5)
    want.backward(g.double())
    unit = {torch.bfloat16: 2.0 ** -9, torch.float16: 2.0 ** -12, torch.float32: 2.0 ** -20}[dtype]
    assert _rel(y, want) < 2 * unit
    for leaf, ref in zip(leaves, wide):
        assert _rel(leaf.grad, ref.grad) < 2 * unit, leaf.shape


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("a_mn, b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("m, n, k", [(768, 768, 8000), (300, 264, 4104), (768, 2304, 8008), (3062, 2048, 8192), (257, 8192, 6000)])
def test_gemm_tiles_cut_along_k(m, n, k, a_mn, b_mn, dtype):
    """The last wave's tiles as ranges of k: every epilogue that they can meet, against 64 bits; the sums stay 32 bits wide."""
    from oslo_b200.ops import cuda_ops as co
    torch.manual_seed(m + n)
    m8 = m if not a_mn else -(-m // 8) * 8
    a = torch.randn(*((k, m8) if a_mn else (m8, k)), device="cuda").to(dtype)
    b = (torch.randn(*((k, n) if b_mn else (n, k)), device="cuda") * k ** -0.5).to(dtype)
    bias, aux = torch.randn(n, device="cuda").to(dtype), torch.randn(m8, n, device="cuda").to(dtype)
    z = (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t())
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    out = aux.clone()
    pre = torch.empty_like(aux)
    g = torch.nn.functional.gelu
    for got, want in ((co.gemm(a, b, a_mn, b_mn), z),
                      (co.gemm(a, b, a_mn, b_mn, bias=bias, aux=aux, flags=co.FLAG_BIAS | co.FLAG_RESIDUAL), z + bias.double() + aux.double()),
                      (co.gemm(a, b, a_mn, b_mn, out=out, flags=co.FLAG_ACCUMULATE), z + aux.double()),
                      (co.gemm(a, b, a_mn, b_mn, bias=bias, aux_out=pre, flags=co.FLAG_BIAS | co.FLAG_GELU | co.FLAG_SAVE_PREACT),
                       g(z + bias.double(), approximate="tanh")), (pre, z + bias.double())):
        assert _rel(got, want) <= eps             # one rounding; GeLU's tanh is good to 2^-11
    y = co.gemm(a, b, a_mn, b_mn, flags=co.FLAG_OUT_FP32)
    assert _rel(y, z) <= 1e-5                     # 32-bit sums of k products: sqrt(8192) roundings of 2^-24, twice over


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n, vocab, width, same", [(1, 5, 8, 0), (129, 50257, 768, 0), (4000, 300, 1032, 0), (5000, 1000, 2048, 3000), (8192, 50400, 4096, 0)])
def test_embedding_gradient_by_rows(n, vocab, width, same, dtype):
    """Sums in 32 bits and one rounding, ids repeated a few times, and one that fills more than a block's list."""
    from oslo_b200.ops import cuda_ops as co
    torch.manual_seed(n)
    ids = torch.randint(0, vocab, (n,), device="cuda")
    ids[torch.randperm(n, device="cuda")[:same]] = vocab // 2
    w = torch.randn(vocab, width, device="cuda").to(dtype).requires_grad_()
    dy = torch.randn(n, width, device="cuda").to(dtype)
    out = co.embedding(ids.view(1, -1), w)
    assert torch.equal(out[0], w.detach()[ids])
    g, = torch.autograd.grad(out, w, dy[None])
    want = torch.zeros(vocab, width, device="cuda", dtype=torch.float64).index_add_(0, ids, dy.double())
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert (g.double() - want).abs().max() <= eps * want.abs().max() + 1e-6 * max(same, 1)    # the second term: 32-bit sums of `same` rows
    assert _rel(g, want) <= eps and not g[torch.bincount(ids, minlength=vocab) == 0].any()
    held = torch.randn(vocab, width, device="cuda").to(dtype)
    w.grad, w._oslo_accum_grad = held.clone(), True
    co.embedding(ids.view(1, -1), w).backward(dy[None])
    assert _rel(w.grad, held.double() + want) <= eps


def _time(call, repeats=20):
    """Median device time of a call, us."""
    for _ in range(3):
        call()
    marks = [torch.cuda.Event(enable_timing=True) for _ in range(repeats + 1)]
    marks[0].record()
    for mark in marks[1:]:
        call()
        mark.record()
    torch.cuda.synchronize()
    return sorted(a.elapsed_time(b) * 1e3 for a, b in zip(marks, marks[1:]))[repeats // 2]


@pytest.mark.parametrize("n, width", [(8000, 768), (7108, 2048)])
@pytest.mark.parametrize("kind", ["one pad id for half", "two type ids"])
def test_embedding_gradient_of_ids_that_fill_a_batch(n, width, kind):
    """Values at every place where an id can start and end in the ordered list, and no slower than three times a batch of all kinds of
    ids (one block that adds up all rows of an id took fifty times that)."""
    from oslo_b200.ops import cuda_ops as co
    torch.manual_seed(n)
    vocab = 50257
    ids = torch.randint(0, vocab, (n,), device="cuda")
    dy = torch.randn(n, width, device="cuda").bfloat16()
    g = torch.zeros(vocab, width, device="cuda", dtype=torch.bfloat16)
    mixed = _time(lambda: co._ext().embedding_grad_(g, ids, dy))
    if kind == "two type ids":
        ids = (torch.arange(n, device="cuda") % 1000 > 500).long() * 7
    else:
        ids[torch.rand(n, device="cuda") < 0.5] = vocab - 1
    same = _time(lambda: co._ext().embedding_grad_(g, ids, dy))
    assert same < 3 * mixed + 20, (same, mixed)
    g.zero_()
    co._ext().embedding_grad_(g, ids, dy)
    want = torch.zeros(vocab, width, device="cuda", dtype=torch.float64).index_add_(0, ids, dy.double())
    assert _rel(g, want) <= 2.0 ** -8
    first = g.clone()
    g.zero_()
    co._ext().embedding_grad_(g, ids, dy)
    assert torch.equal(g, first)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 65, 1000, 2049, 32768])
def test_embedding_gradient_at_the_edges_of_its_chunks(n):
    """Ids whose rows end, start and go on at chunks of 32 ordered tokens; ids outside the vocabulary are skipped."""
    from oslo_b200.ops import cuda_ops as co
    torch.manual_seed(n)
    dy = torch.randn(n, 264, device="cuda").half()
    for ids in (torch.zeros(n), torch.arange(n) // 32, (torch.arange(n) + 16) // 32, torch.arange(n) // 96, torch.arange(n).flip(0) // 33,
                torch.arange(n) % 5, torch.arange(n) % 40 - 3):
        ids = ids.long().cuda()
        vocab = int(ids.max().clamp_min(0)) + 1 if int(ids.min()) >= 0 else 30
        g = torch.zeros(vocab, 264, device="cuda").half()
        co._ext().embedding_grad_(g, ids, dy)
        ok = (ids >= 0) & (ids < vocab)
        want = torch.zeros(vocab, 264, device="cuda", dtype=torch.float64).index_add_(0, ids[ok], dy[ok].double())
        assert (g.double() - want).abs().max() <= 2.0 ** -11 * want.abs().max() + 1e-5 * n ** 0.5      # one rounding; 32-bit sums of up to n rows
    co.reset_device_error(dy)


@pytest.mark.parametrize("cols", [8, 64, 640, 1344, 2056])
def test_gated_units_of_narrow_rows(cols):
    """The same number of values in rows of any width: all of a block's threads have work (one row per block of 256 threads left 248 of
    them idle at 64 columns)."""
    from oslo_b200.ops import cuda_ops as co
    from oslo_b200.ops import reference as ref
    rows = 8192 * 5120 // cols
    mk = lambda r, c: torch.randn(r, c, device="cuda").bfloat16()        # noqa: E731
    a, b, wa, wb = mk(rows, cols), mk(rows, cols), mk(8192, 5120), mk(8192, 5120)
    assert _time(lambda: co.silu_mul(a, b)) < 1.6 * _time(lambda: co.silu_mul(wa, wb)) + 10
    assert _rel(co.silu_mul(a[:999], b[:999]), ref.silu_mul(a[:999].double(), b[:999].double())) <= 2.0 ** -8


def test_embedding_gradient_by_every_way_of_asking():
    """``torch.autograd.grad``, ``backward(inputs=...)``, second derivatives, function transforms and forward mode, of a weight whose
    gradient lives in a flat buffer: what the library's lookup gives (sums of a few 16-bit values; exact in 32 bits, rounded once)."""
    from oslo_b200.parallel.layers import Embedding
    torch.manual_seed(0)
    ids, other = torch.randint(0, 50, (4, 33), device="cuda"), torch.randn(64, device="cuda").bfloat16().requires_grad_()
    emb = Embedding(50, 64).to("cuda", torch.bfloat16)
    emb.oslo_fused = True
    w = emb.weight
    w.grad, w._oslo_accum_grad = torch.ones_like(w), True
    plain = torch.nn.functional.embedding
    loss = lambda x: (x.float() * other.float()).square().sum()        # noqa: E731
    want, = torch.autograd.grad(loss(plain(ids, w)), w)
    got, = torch.autograd.grad(loss(emb(ids)), w)
    assert _rel(got, want) <= 2.0 ** -8 and torch.equal(w.grad, torch.ones_like(w))
    loss(emb(ids)).backward(inputs=[other])
    assert torch.equal(w.grad, torch.ones_like(w))
    second = []
    for look in (lambda: emb(ids), lambda: plain(ids, w)):
        g, = torch.autograd.grad(loss(look()), w, create_graph=True)
        second.append(torch.autograd.grad(g.float().square().sum(), other)[0])
    assert _rel(*second) <= 2.0 ** -7
    got = torch.func.grad(lambda p: loss(torch.func.functional_call(emb, {"weight": p}, (ids,))))(w)
    assert _rel(got, want) <= 2.0 ** -8
    assert torch.equal(torch.func.vmap(emb)(ids), plain(ids, w))
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(w.detach().requires_grad_(), torch.ones_like(w))
        tangent = torch.autograd.forward_ad.unpack_dual(torch.func.functional_call(emb, {"weight": dual}, (ids,))).tangent
    assert torch.equal(tangent, torch.ones_like(tangent))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows", [296, 297, 1000])
@pytest.mark.parametrize("cols, top", [(512, 1), (520, 3), (1024, 2), (2048, 3), (2056, 2), (4096, 5), (4104, 3)])
def test_branch_join_rows(rows, cols, top, dtype):
    """Both sides of the rule for whole rows in registers, against 64 bits: branches with and without a norm, gathered and scaled ones."""
    from oslo_b200.ops import cuda_ops as co
    from oslo_b200.ops.reference import Branch
    torch.manual_seed(rows + cols)
    mk = lambda *s: torch.randn(*s, device="cuda").to(dtype)  # noqa: E731
    x, w1, w2, wn = torch.randn(rows, cols, device="cuda"), mk(cols), mk(cols), mk(cols)
    slots = torch.randperm(rows * top + 5, device="cuda")[:rows * top].int().view(rows, top)
    many, one, normed = mk(rows * top + 5, cols), mk(rows, cols + 8)[:, :cols], mk(rows, cols)
    got, copies = co.branch_join(x, [Branch(many, slots=slots, top=top), Branch(one), Branch(normed, weight=wn, normed=True)], 0.5, 1e-5, [w1, w2])
    d = normed.double()
    z = x.double() + 0.5 * (many.double()[slots.long()].sum(1) + one.double() + d * torch.rsqrt(d.square().mean(-1, keepdim=True) + 1e-5) * wn.double())
    r = torch.rsqrt(z.square().mean(-1, keepdim=True) + 1e-5)
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert _rel(got, z) <= 1e-6 and _rel(copies[0], z * r * w1.double()) <= eps and _rel(copies[1], z * r * w2.double()) <= eps

"""The decode step's kernels at the edges of their tiles: products of 1 to 64 rows, and attention that appends the new token itself."""
import pytest
import torch

import oslo_b200 as ob

pytestmark = pytest.mark.gpu
EPS = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}


def _close(y, ref, dtype):
    """One rounding to 16 bits (half a unit of ``EPS`` per value) and 32-bit sums; the rest covers a row's GeLU by tanh.approx."""
    assert torch.isfinite(y).all()
    assert (y.double() - ref).norm() <= 1.5 * EPS[dtype] * ref.norm()
    assert (y.double() - ref).abs().max() <= 4 * EPS[dtype] * ref.abs().max()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kn", [False, True])
@pytest.mark.parametrize("m", [1, 2, 3, 5, 8, 9, 16, 17, 31, 33, 64])
@pytest.mark.parametrize("k1, k2, n", [(8, 0, 8), (40, 0, 72), (768, 0, 2304), (256, 1032, 264), (4104, 0, 1000), (64, 0, 50264)])
def test_few_rows(dtype, kn, m, k1, k2, n):
    from oslo_b200.ops import cuda_ops
    ext = cuda_ops._ext()
    torch.manual_seed(m * 7 + k1 + n)
    mk = lambda *s: torch.randn(*s, device="cuda").to(dtype)  # noqa: E731
    x1, x2, bias, res = mk(m, k1 + 8)[:, :k1], (mk(m, k2) if k2 else None), mk(n), mk(m, n)
    w = mk(k1 + k2, n) if kn else mk(n, k1 + k2)
    x = x1 if x2 is None else torch.cat([x1, x2], 1)
    z = x.double() @ (w.double() if kn else w.double().t())
    y = ext.few_rows(x1, x2, [w], int(kn), bias, n // 2, res)
    z = z + bias.double()
    z[:, n // 2:] = torch.nn.functional.gelu(z[:, n // 2:], approximate="tanh")
    _close(y, z + res.double(), dtype)
    if not kn and k2 == 0:
        _close(ext.few_rows(x1, None, [w, w.flip(0).contiguous()], 0, None, -1), torch.cat([x1.double() @ w.double().t(), x1.double() @ w.flip(0).double().t()], 1), dtype)
        odd = n - 3                                            # columns past the end belong to nobody
        _close(ext.few_rows(x1, None, [w[:odd]], 0, bias[:odd], -1), x1.double() @ w[:odd].double().t() + bias[:odd].double(), dtype)
    if m <= 8 and k2 == 0 and m * k1 <= 8192:
        ln = torch.nn.LayerNorm(k1).to("cuda", dtype)
        with torch.no_grad():
            ln.weight.normal_(1, 0.1), ln.bias.normal_(0, 0.1)
            h = torch.nn.functional.layer_norm(x1.double(), (k1,), ln.weight.double(), ln.bias.double(), ln.eps)
            y = ext.few_rows(x1, None, [w], int(kn), None, -1, None, ln.weight, ln.bias, ln.eps)
        # the normalised input is rounded to 16 bits, as the LayerNorm kernel rounds it
        ref = h @ (w.double() if kn else w.double().t())
        bound = 1.5 * EPS[dtype] * (h.norm() * w.double().norm() / (k1 * n) ** 0.5 * n ** 0.5 + ref.norm())
        assert torch.isfinite(y).all() and (y.double() - ref).norm() <= bound


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kn, m, k1, k2, n", [(0, 1, 8200, 8184, 4100), (0, 1, 16384, 0, 4098), (0, 1, 2056, 0, 2368), (0, 1, 2048, 8, 2372), (0, 2, 16392, 0, 4100),
                                              (1, 1, 4104, 0, 2048), (1, 8, 4096, 8, 2056), (1, 3, 4088, 16, 2048), (1, 5, 3072, 0, 2048), (1, 5, 3080, 0, 2048)])
def test_few_rows_on_both_sides_of_the_rules_for_large_weights(dtype, kn, m, k1, k2, n):
    """One row with few outputs or 64 M values and more; [in, out] weights below and above 6 M values, their k from one and two inputs."""
    from oslo_b200.ops import cuda_ops
    torch.manual_seed(k1 + n)
    mk = lambda *s: torch.randn(*s, device="cuda").to(dtype)  # noqa: E731
    x1, x2, bias, res = mk(m, k1), (mk(m, k2) if k2 else None), mk(n), mk(m, n)
    w = mk(k1 + k2, n) if kn else mk(n, k1 + k2)
    x = x1 if x2 is None else torch.cat([x1, x2], 1)
    z = x.double() @ (w.double() if kn else w.double().t()) + bias.double()
    z[:, n // 2:] = torch.nn.functional.gelu(z[:, n // 2:], approximate="tanh")
    _close(cuda_ops._ext().few_rows(x1, x2, [w], kn, bias, n // 2, res), z + res.double(), dtype)


@pytest.mark.parametrize("rows", [1, 3, 9])
@pytest.mark.parametrize("n", [40, 37, 1])
def test_linear_of_operands_at_odd_addresses(rows, n):
    """Views that start between 16-byte boundaries, or single rows cut out of longer odd ones, are copied."""
    from oslo_b200.ops import cuda_ops
    torch.manual_seed(n)
    buf = torch.randn(64 * 64 + 64 * 67, device="cuda").bfloat16()
    weights = [buf[3:3 + n * 64].view(n, 64), buf[:n * 64].view(n, 64)]
    inputs = [buf[5:5 + rows * 64].view(rows, 64), buf[:rows * 67].view(rows, 67)[:, :64], buf[8:8 + rows * 64].view(rows, 64)]
    with torch.no_grad():
        for w in weights:
            for x in inputs:
                _close(ob.ops.linear(x, w), x.double() @ w.double().t(), torch.bfloat16)
                res = buf[:2 * rows * n:2].view(n, rows).t()
                y = cuda_ops.linear(x, w, None, False, None, res)
                _close(y, x.double() @ w.double().t() + res.double(), torch.bfloat16)


@pytest.mark.parametrize("m", [9, 64])
@pytest.mark.parametrize("k, n", [(1024, 1032), (2048, 136)])
def test_several_weights_of_any_width_are_not_copied(m, k, n):
    """Widths that are no multiple of the tile's 128 columns: no memory but the result's."""
    from oslo_b200.ops import cuda_ops
    torch.manual_seed(n)
    mk = lambda *s: torch.randn(*s, device="cuda").bfloat16()  # noqa: E731
    x, ws, bias, res = mk(m, k), [mk(n, k) for _ in range(3)], mk(3 * n), mk(m, 3 * n)
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    y = cuda_ops._ext().few_rows(x, None, ws, 0, bias, n + 40, res)
    assert torch.cuda.max_memory_allocated() - before < 2 * n * k * 2
    z = torch.cat([x.double() @ w.double().t() for w in ws], 1) + bias.double()
    z[:, n + 40:] = torch.nn.functional.gelu(z[:, n + 40:], approximate="tanh")
    _close(y, z + res.double(), torch.bfloat16)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kn", [False, True])
@pytest.mark.parametrize("m", [64, 65, 128])
@pytest.mark.parametrize("k, n", [(64, 72), (60, 72), (64, 68), (4104, 1000)])
@pytest.mark.parametrize("gelu_from", [-1, 0, 24])
def test_small_products_of_up_to_128_rows(dtype, kn, m, k, n, gelu_from):
    """The operator on operands whose rows are aligned, whatever their sizes."""
    from oslo_b200.ops import cuda_ops
    torch.manual_seed(m + k + n)
    mk = lambda r, c: torch.randn(r, -(-c // 8) * 8, device="cuda").to(dtype)[:, :c]  # noqa: E731
    a, b, bias = mk(m, k), mk(k, n) if kn else mk(n, k), torch.randn(n, device="cuda").to(dtype)
    z = a.double() @ (b.double() if kn else b.double().t()) + bias.double()
    if gelu_from >= 0:
        z[:, gelu_from:] = torch.nn.functional.gelu(z[:, gelu_from:], approximate="tanh")
    _close(cuda_ops._ext().gemm_small_m(a, b, int(kn), bias, gelu_from), z, dtype)


@pytest.mark.parametrize("rows", [1, 4, 5, 8, 9])
@pytest.mark.parametrize("layout", ["plain", "transposed weight", "sliced x", "odd x"])
def test_stacked_products_of_any_layout(rows, layout):
    from oslo_b200.ops import cuda_ops
    torch.manual_seed(rows)
    parts, k, n = 3, 64, 40
    mk = lambda *s: torch.randn(*s, device="cuda").bfloat16()  # noqa: E731
    w = mk(parts, k, n).transpose(1, 2) if layout == "transposed weight" else mk(parts, n, k)
    x = mk(parts, rows, k)
    if layout == "sliced x":
        x = mk(parts, rows, 2 * k)[:, :, k:]
    elif layout == "odd x":
        x = mk(parts, rows, k + 3)[:, :, 1:k + 1]
    for i, y in enumerate(cuda_ops.stacked_linear(x, w)):
        _close(y, x[i].double() @ w[i].double().t(), torch.bfloat16)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("d, rotary", [(8, 0), (32, 8), (64, 0), (80, 32), (128, 64), (256, 64), (256, 0)])
@pytest.mark.parametrize("b, h, t, at, window", [(1, 3, 1, 0, 0), (2, 12, 180, 173, 0), (8, 16, 512, 300, 0), (1, 16, 2048, 2047, 0), (3, 5, 700, 690, 256),
                                                 (40, 16, 96, 33, 17)])
def test_decode_step_attention(dtype, d, rotary, b, h, t, at, window):
    """Append, rotary and attention in one kernel against the three separate statements."""
    from oslo_b200.ops import cuda_ops
    torch.manual_seed(d + t + b)
    qkv = torch.randn(b, 3 * h * d + 8, device="cuda").to(dtype)
    q, k, v = (qkv[:, i * h * d:(i + 1) * h * d].unflatten(1, (h, d)) for i in range(3))
    kc, vc = (torch.randn(b, h, t, d, device="cuda").to(dtype) for _ in range(2))
    kc[:, :, at:], vc[:, :, at:] = float("nan"), float("nan")   # what lies behind the new token is not read
    lengths = torch.full((b,), at + 1, device="cuda", dtype=torch.int32)
    index = torch.full((1,), at, device="cuda", dtype=torch.long)
    k2, v2 = kc.clone(), vc.clone()
    out = cuda_ops.decode_step_attention(q, k, v, k2, v2, lengths, lengths - 1, index, d ** -0.5, window or None, rotary)
    if rotary:
        pos = (lengths - 1).long()[:, None]
        rot = lambda z: ob.ops.rotary_interleaved(z[:, None], pos, rotary)[:, 0]  # noqa: E731
        q, k = rot(q), rot(k)
    kc[:, :, at], vc[:, :, at] = k, v
    tol = dict(atol=2 * EPS[dtype], rtol=4 * EPS[dtype])        # the prefill's rotary kernel may round the other way
    torch.testing.assert_close(k2[:, :, :at + 1], kc[:, :, :at + 1], **tol)
    assert torch.equal(v2[:, :, :at + 1], vc[:, :, :at + 1]) and torch.isnan(v2[:, :, at + 1:]).all()
    lo = max(0, at + 1 - window) if window else 0
    s = torch.einsum("bhd,bhtd->bht", q.double(), k2[:, :, lo:at + 1].double()) * d ** -0.5
    ref = torch.einsum("bht,bhtd->bhd", s.softmax(-1), v2[:, :, lo:at + 1].double())
    torch.testing.assert_close(out.double(), ref, atol=3 * EPS[dtype], rtol=3 * EPS[dtype])
    torch.testing.assert_close(cuda_ops.decode_attention(q, k2, v2, lengths, d ** -0.5, window or None).double(), ref, atol=3 * EPS[dtype], rtol=3 * EPS[dtype])


@pytest.mark.parametrize("kind", ["gpt2", "gpt_neo", "gptj"])
def test_a_step_replayed_past_the_end_of_the_cache_is_refused(kind):
    """A captured step of the user's own, one replay too many: no finite logits, nothing written, and the device's error word says so."""
    from oslo_b200.models.common import StaticKVCache
    from oslo_b200.ops import cuda_ops
    if kind == "gpt2":
        model = ob.GPT2LMHeadModel(ob.GPT2Config(vocab_size=64, n_positions=64, n_embd=64, n_layer=2, n_head=2))
    elif kind == "gpt_neo":
        model = ob.GPTNeoForCausalLM(ob.GPTNeoConfig(vocab_size=64, max_position_embeddings=64, hidden_size=64, num_layers=2, num_heads=2,
                                                     window_size=4, attention_types=[[["global", "local"], 1]]))
    else:
        model = ob.GPTJForCausalLM(ob.GPTJConfig(vocab_size=64, n_positions=64, n_embd=64, n_layer=2, n_head=2, rotary_dim=16))
    model = model.to("cuda", torch.bfloat16).fuse().eval()
    ids, cache = torch.zeros(3, 6, dtype=torch.long, device="cuda"), StaticKVCache(8)
    step = lambda: model(input_ids=ids[:, :1], past_key_values=cache, position_ids=cache.lengths_dev.long()[:, None], use_cache=True).logits  # noqa: E731
    with torch.no_grad():
        model(input_ids=ids, past_key_values=cache, use_cache=True)
        cache.use_device_positions()
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            step()                                    # the first of two places
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = step()
    cuda_ops.reset_device_error(ids)
    graph.replay()
    assert torch.isfinite(out).all() and cuda_ops.device_error_code(ids) == 0
    held = [t.clone() for t in (*cache.k.values(), *cache.v.values())]
    graph.replay()
    assert not torch.isfinite(out).any() and cuda_ops.device_error_code(ids) == 6
    assert all(torch.equal(a, b) for a, b in zip(held, (*cache.k.values(), *cache.v.values())))
    cuda_ops.reset_device_error(ids)


@pytest.mark.parametrize("b, h, s, d, t, start", [(1, 1, 1, 8, 1, 0), (2, 3, 17, 64, 40, 5), (4, 16, 200, 256, 210, 10), (3, 5, 333, 80, 333, 0)])
def test_prompt_append(b, h, s, d, t, start):
    """Keys and values of a prompt land where slice copies put them, from slices of joint rows and from contiguous tensors."""
    from oslo_b200.ops import cuda_ops
    for k, v in (torch.randn(b, s, 2, h, d, device="cuda").bfloat16().permute(2, 0, 3, 1, 4).unbind(0),
                 (torch.randn(b, h, s, d, device="cuda").bfloat16(), torch.randn(b, s, h, d, device="cuda").bfloat16().transpose(1, 2))):
        kc, vc = (torch.randn(b, h, t, d, device="cuda").bfloat16() for _ in range(2))
        k2, v2 = kc.clone(), vc.clone()
        assert cuda_ops.prompt_append_ok(k, v, k2, v2)
        cuda_ops.prompt_append(k, v, k2, v2, start)
        kc[:, :, start:start + s], vc[:, :, start:start + s] = k, v
        assert torch.equal(k2, kc) and torch.equal(v2, vc)


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("b, s, h, d, window", [(2, 65, 3, 64, 0), (1, 300, 2, 128, 40)])
def test_packed_attention_is_the_split_one(b, s, h, d, window, masked):
    from oslo_b200.ops import cuda_ops
    torch.manual_seed(s)
    qkv = torch.randn(b, s, 3 * h * d, device="cuda").bfloat16().requires_grad_()
    mask = (torch.arange(s, device="cuda") < s - 7).long().expand(b, s) if masked else None
    g = torch.randn(b, h, s, d, device="cuda").bfloat16()
    a = cuda_ops.packed_attention(qkv, h, window or None, d ** -0.5, mask)
    ga, = torch.autograd.grad(a, qkv, g)
    q, k, v = (x.unflatten(-1, (h, d)).transpose(1, 2) for x in qkv.split(h * d, dim=2))
    c = cuda_ops.flash_attention(q, k, v, True, window or None, d ** -0.5, mask)
    gc, = torch.autograd.grad(c, qkv, g)
    assert torch.equal(a, c) and torch.equal(ga, gc)


@pytest.mark.parametrize("reversed_", [False, True])
def test_fused_mlp_layouts(reversed_):
    """Both weight layouts of the two-layer node against 64-bit autograd: one rounding of each of four 16-bit intermediates."""
    from oslo_b200.ops import cuda_ops
    torch.manual_seed(1)
    n, w, f = 200, 72, 264
    p = [torch.randn(*s, device="cuda") * sc for s, sc in (((n, w), 1), ((f, w), 0.1), ((f,), 0.1), ((w, f), 0.1), ((w,), 0.1), ((n, w), 1))]
    p = [x.bfloat16().requires_grad_() for x in p]
    x, w1, b1, w2, b2, r = p
    g = torch.randn(n, w, device="cuda").bfloat16()
    a, c = (w1.t().contiguous(), w2.t().contiguous()) if reversed_ else (w1, w2)
    y = cuda_ops.fused_mlp(x, a, b1, c, b2, r, reversed_)
    got = torch.autograd.grad(y, p, g)
    d = [t.detach().double().requires_grad_() for t in p]
    ref = torch.nn.functional.gelu(d[0] @ d[1].t() + d[2], approximate="tanh") @ d[3].t() + d[4] + d[5]
    want = torch.autograd.grad(ref, d, g.double())
    for have, need in zip((y, *got), (ref, *want)):
        assert (have.double() - need).norm() <= 4 * 2.0 ** -8 * need.norm()

"""When a block of GPT-2 or GPT-Neo may compute what its modules compute without calling them, or call them with more than their
input: on fake CUDA tensors, whose every Python branch runs. ``called`` records the calls of the layers' ``forward``."""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

import oslo_b200 as ob
from oslo_b200 import ops
from oslo_b200.parallel import layers as L

from .test_fake_cuda import _model

KINDS = ["gpt2", "gpt_neo"]


@pytest.fixture
def kernels(monkeypatch):
    if ops.load_ext() is None:
        pytest.skip("extension not built")
    monkeypatch.setattr(ops, "kernels_available", lambda: True)


@pytest.fixture
def called(monkeypatch):
    seen = {}
    for cls in (L.Conv1D, L.Linear):
        def forward(self, x, activation=None, residual=None, _old=cls.forward):
            seen[id(self)] = residual is not None
            return _old(self, x, activation, residual)
        monkeypatch.setattr(cls, "forward", forward)
    return seen


def _fused(kind):
    cls, cfg = _model(kind)
    if kind == "gpt2":
        cfg.resid_pdrop = 0.0
    with torch.device("cuda"):
        model = cls._from_config(cfg, torch_dtype=torch.bfloat16)
    return model.fuse()


def _parts(model, kind):
    block = model.transformer.h[0]
    attn = block.attn if kind == "gpt2" else block.attn.attention
    return block, attn, (attn.c_proj if kind == "gpt2" else attn.out_proj)


def _ids():
    return torch.zeros(2, 64, dtype=torch.long, device="cuda")


@pytest.mark.parametrize("kind", KINDS)
def test_layers_nobody_listens_to_are_not_called(kernels, called, kind):
    with FakeTensorMode():
        model = _fused(kind).train()
        block, attn, out_proj = _parts(model, kind)
        model(input_ids=_ids())
        assert id(block.mlp.c_fc) not in called and called[id(out_proj)]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("register", ["register_full_backward_hook", "register_full_backward_pre_hook"])
@pytest.mark.parametrize("name", ["mlp", "mlp.c_fc", "mlp.c_proj", "attn.attention.q_proj"])
def test_a_backward_hook_has_its_module_called(kernels, called, kind, register, name):
    with FakeTensorMode():
        model = _fused(kind).train()
        block, _, _ = _parts(model, kind)
        if name.startswith("attn.attention") and kind == "gpt2":
            pytest.skip("GPT-Neo's layers")
        getattr(block.get_submodule(name), register)(lambda *a: None)
        model(input_ids=_ids())
        layer = block.mlp.c_fc if name == "mlp" else block.get_submodule(name)
        assert id(layer) in called


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("register", ["register_module_full_backward_hook", "register_module_full_backward_pre_hook"])
def test_a_global_backward_hook_has_all_modules_called(kernels, called, kind, register):
    with FakeTensorMode():
        model = _fused(kind).train()
        block, _, _ = _parts(model, kind)
        handle = getattr(torch.nn.modules.module, register)(lambda *a: None)
        try:
            model(input_ids=_ids())
        finally:
            handle.remove()
        assert id(block.mlp.c_fc) in called


@pytest.mark.parametrize("train", [True, False])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("where", ["attn", "attention", "out_proj"])
def test_a_hook_on_attention_gets_the_attention_alone(kernels, called, kind, where, train):
    """The residual stream is not added inside modules whose output somebody takes or replaces."""
    with FakeTensorMode():
        model = _fused(kind).train(train)
        block, attn, out_proj = _parts(model, kind)
        {"attn": block.attn, "attention": attn, "out_proj": out_proj}[where].register_forward_hook(lambda *a: None)
        with torch.set_grad_enabled(train):
            model(input_ids=_ids())
        assert called[id(out_proj)] is False


class _OwnAttention(torch.nn.Module):
    """A user's attention: its own signature, none of the attributes of the family's."""

    def forward(self, hidden_states, layer_past=None, attention_mask=None, position_ids=None, head_mask=None, use_cache=False,
                output_attentions=False, cache=None, layer_id=0, seq_shape=None):
        return 2 * hidden_states, None, None


@pytest.mark.parametrize("device", ["cpu", "cuda"])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("part", ["mlp", "attn"])
def test_a_part_of_the_users_own_is_called(kernels, kind, device, part):
    from oslo_b200.models.common import StaticKVCache
    cls, cfg = _model(kind)
    with FakeTensorMode():
        with torch.device(device):
            model = cls._from_config(cfg, torch_dtype=torch.bfloat16)
        if device == "cuda":
            model.fuse()
        model.eval()
        for block in model.transformer.h:
            setattr(block, part, torch.nn.SiLU() if part == "mlp" else _OwnAttention())
        ids = _ids().to(device)
        for kw in ({}, {"past_key_values": StaticKVCache(100)})[:2 if part == "mlp" else 1]:     # this attention fills no cache
            with torch.no_grad():
                assert model(input_ids=ids, use_cache=bool(kw), **kw).logits.shape[:2] == (2, 64)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("how", ["mlp class", "mlp forward", "c_fc forward", "attention class", "attention forward", "out_proj forward"])
def test_overridden_modules_are_called(kernels, called, kind, how):
    """Subclasses of the family's modules, and modules with a ``forward`` of their own, in a prompt and in a step on device positions."""
    from oslo_b200.models.common import StaticKVCache
    with FakeTensorMode():
        model = _fused(kind).eval()
        seen = []
        for block in model.transformer.h:
            attn = block.attn if kind == "gpt2" else block.attn.attention
            out_proj = attn.c_proj if kind == "gpt2" else attn.out_proj
            target = {"mlp": block.mlp, "c_fc": block.mlp.c_fc, "attention": attn, "out_proj": out_proj}[how.split()[0]]
            if how.endswith("class"):
                base = type(target)

                def forward(self, x, _base=base, **kw):
                    seen.append(kw.get("residual"))
                    return _base.forward(self, x, **kw)
                target.__class__ = type("Own", (base,), {"forward": forward})
            else:
                def forward(x, _old=target.forward, **kw):
                    seen.append(kw.get("residual"))
                    return _old(x, **kw)
                target.forward = forward
        with torch.no_grad():
            cache = StaticKVCache(100)
            model(input_ids=_ids(), past_key_values=cache, use_cache=True)
            assert len(seen) == len(model.transformer.h)
            cache.use_device_positions()
            model(input_ids=_ids()[:, :1], past_key_values=cache, use_cache=True)
        assert len(seen) == 2 * len(model.transformer.h) and all(r is None for r in seen)


@pytest.mark.parametrize("step", [False, True])
def test_gptj_attention_and_mlp_get_the_normed_stream(kernels, monkeypatch, step):
    """Few rows whose q, k, v and first MLP layer are one product, outside the whole-block step: attention and MLP are called, and
    with what the norm returned."""
    from oslo_b200.models.common import StaticKVCache
    normed, got = [], []
    old = L.LayerNorm.forward
    monkeypatch.setattr(L.LayerNorm, "forward", lambda self, x: normed.append(old(self, x)) or normed[-1])
    cls, cfg = _model("gptj")
    with FakeTensorMode():
        with torch.device("cuda"):
            model = cls._from_config(cfg, torch_dtype=torch.bfloat16)
        model.fuse().eval()
        ids, cache = torch.zeros(2, 4 if not step else 1, dtype=torch.long, device="cuda"), StaticKVCache(100)
        with torch.no_grad():
            if step:       # a step whose keys are masked
                model(input_ids=ids, past_key_values=cache, use_cache=True)
                cache.use_device_positions()
            for block in model.transformer.h:
                for m in (block.attn, block.mlp):
                    m.register_forward_pre_hook(lambda m, args: got.append(args[0]))
            normed.clear()
            model(input_ids=ids, past_key_values=cache, use_cache=True,
                  **({"attention_mask": torch.ones(2, 2, dtype=torch.long, device="cuda")} if step else {}))
    assert len(got) == 4 and all(any(g is n for n in normed) for g in got)


@pytest.mark.parametrize("kind", KINDS)
def test_without_the_extension_the_fallback_runs(monkeypatch, kind):
    """``OSLO_B200_ALLOW_FALLBACK=1``: prompt, step on device positions and training through the PyTorch statements."""
    from oslo_b200.models.common import StaticKVCache
    from oslo_b200.ops import cuda_ops

    def load_ext(required=False):
        if required:
            raise RuntimeError("CUDA extension unavailable")
    monkeypatch.setattr(ops, "load_ext", load_ext)
    monkeypatch.setattr(cuda_ops, "load_ext", load_ext)
    monkeypatch.setenv("OSLO_B200_ALLOW_FALLBACK", "1")
    with FakeTensorMode():
        model = _fused(kind).eval()
        cache = StaticKVCache(100)
        with torch.no_grad():
            model(input_ids=_ids(), past_key_values=cache, use_cache=True)
            cache.use_device_positions()
            assert model(input_ids=_ids()[:, :1], past_key_values=cache, use_cache=True).logits.shape[:2] == (2, 1)
        assert model.train()(input_ids=_ids(), labels=_ids()).loss.shape == ()
        x = torch.zeros(2, 1, 512, device="cuda", dtype=torch.bfloat16)
        assert model.transformer.h[0].mlp.c_proj(x.new_zeros(2, 100, 2048), residual=x.new_zeros(2, 100, 512)).shape == (2, 100, 512)


@pytest.mark.parametrize("rows", [4, 5, 64])
@pytest.mark.parametrize("rank", [0, 1])
def test_gptj_tensor_parallel_step_adds_the_residual_after_the_reduction(kernels, monkeypatch, rows, rank):
    """More than 4 rows: the parts that are summed over the ranks are products alone."""
    from types import SimpleNamespace

    from oslo_b200.models.common import StaticKVCache
    from oslo_b200.ops import cuda_ops
    products, reduced = [], []
    old = cuda_ops.gemv_two_inputs
    monkeypatch.setattr(cuda_ops, "gemv_two_inputs", lambda *a: products.append((a[3], a[4], old(*a))) or products[-1][2])
    mpu = SimpleNamespace(tp=2, tp_rank=rank, _reduce=lambda z: reduced.append(z) or z)
    cls, cfg = _model("gptj")
    with FakeTensorMode():
        with torch.device("cuda"):
            model = cls._from_config(cfg, torch_dtype=torch.bfloat16)
        model.fuse().eval()
        ids, cache = torch.zeros(rows, 8, dtype=torch.long, device="cuda"), StaticKVCache(100)
        with torch.no_grad():
            model(input_ids=ids, past_key_values=cache, use_cache=True)
            cache.use_device_positions()
            for block in model.transformer.h:
                block.attn.out_proj.mpu = mpu
            assert model(input_ids=ids[:, :1], past_key_values=cache, use_cache=True).logits.shape[0] == rows
    assert len(products) == len(reduced) == len(model.transformer.h)
    inside = rows <= 4 and rank == 0
    for (bias, residual, y), z in zip(products, reduced):
        assert (bias is not None) == inside and (residual is not None) == inside and z is y


def _reached(out):
    """The leaves that a backward pass from ``out`` reaches through nodes that have one."""
    seen, keep, stack, leaves = set(), [], [out.grad_fn], []
    while stack:
        node = stack.pop()
        if node is None or id(node) in seen or "NotImplemented" in node.name():
            continue
        seen.add(id(node))
        keep.append(node)
        if hasattr(node, "variable"):
            leaves.append(node.variable)
        stack += [fn for fn, _ in node.next_functions]
    return leaves


@pytest.mark.parametrize("kind", ["gpt2", "gpt_neo", "gptj"])
@pytest.mark.parametrize("which", ["weight", "bias"])
def test_a_step_with_trainable_norms_keeps_their_graph(kernels, kind, which):
    """Frozen layers, norms that learn: a step with gradients enabled is part of the graph."""
    from oslo_b200.models.common import StaticKVCache
    cls, cfg = _model(kind)
    with FakeTensorMode():
        with torch.device("cuda"):
            model = cls._from_config(cfg, torch_dtype=torch.bfloat16)
        model.fuse().eval().requires_grad_(False)
        block = model.transformer.h[0]
        x = torch.zeros(2, 1, 512, dtype=torch.bfloat16, device="cuda")
        cache = StaticKVCache(100)
        with torch.no_grad():
            model(input_ids=_ids(), past_key_values=cache, use_cache=True)
        cache.use_device_positions()
        kw = dict(cache=cache, layer_id=0, use_cache=True, position_ids=torch.full((2, 1), 64, dtype=torch.long, device="cuda"))
        assert not block(x, **kw)[0].requires_grad
        norm = block.ln_1 if kind == "gptj" else block.ln_2       # the one with a way past the attention kernel, which has no backward
        p = getattr(norm, which).requires_grad_(True)
        assert any(leaf is p for leaf in _reached(block(x, **kw)[0]))


@pytest.mark.parametrize("kind", ["gpt2", "gpt_neo", "gptj"])
def test_a_step_with_a_norm_bias_of_another_type(kernels, monkeypatch, kind):
    """No kernel takes such a bias: the norm stays a call of its own."""
    from oslo_b200.models.common import StaticKVCache
    from oslo_b200.ops import cuda_ops
    folded = []
    old = cuda_ops.few_rows
    monkeypatch.setattr(cuda_ops, "few_rows", lambda *a, **k: folded.append(k.get("ln")) or old(*a, **k))
    cls, cfg = _model(kind)
    with FakeTensorMode():
        with torch.device("cuda"):
            model = cls._from_config(cfg, torch_dtype=torch.bfloat16)
        model.fuse().eval().requires_grad_(False)
        cache = StaticKVCache(100)
        model(input_ids=_ids(), past_key_values=cache, use_cache=True)
        cache.use_device_positions()
        block = model.transformer.h[0]
        kw = dict(cache=cache, layer_id=0, use_cache=True, position_ids=torch.full((2, 1), 64, dtype=torch.long, device="cuda"))
        x = torch.zeros(2, 1, 512, dtype=torch.bfloat16, device="cuda")
        folded.clear()
        block(x, **kw)
        assert any(ln is not None for ln in folded)
        norms = [getattr(block, n) for n in ("ln_1", "ln_2") if hasattr(block, n)]
        for ln in norms:
            ln.bias = torch.nn.Parameter(ln.bias.float(), requires_grad=False)
        folded.clear()
        try:
            block(x, **kw)
        except RuntimeError as e:       # the norm's own call may not take it either
            assert "LayerNorm" not in str(e)
        assert not any(ln is not None for ln in folded)

"""What sends a call from the whole-model and whole-module library calls back to the modules, and what the caller sees of them."""

import pytest
import torch
import torch.nn as nn
from torch.nn.modules import module as nn_module

from titanmac_b200 import (BlockSparseAttention, TitanMAC, TitanMACConfig, WindowConfig, WindowedAttention, _native, _stack,
                           _train)

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF16 = torch.bfloat16


def make(block_sparse=False, layers=2, vocab=128, heads=2, dh=64, n_p=3, seed=0, **more):
    cfg = TitanMACConfig(vocab_size=vocab, d_model=heads * dh, n_heads=heads, n_layers=layers, d_ff=3 * heads * dh, max_seq_len=64,
                         window_size=16, n_persistent=n_p, use_block_sparse=block_sparse, block_size=32, **more)
    g = torch.Generator(device=DEV).manual_seed(seed)
    with torch.device(DEV):
        model = TitanMAC(cfg)
    with torch.no_grad():
        for name, prm in model.named_parameters():
            prm.normal_(1.0 if name.endswith("scale") else 0.0, 0.1 if name.endswith(("scale", "bias")) else 0.04, generator=g)
    return model.to(BF16), torch.randint(0, vocab, (2, 30), generator=g, device=DEV)


def module_by_module(monkeypatch):
    monkeypatch.setattr(_stack, "table_of", lambda *a, **k: None)
    monkeypatch.setattr(_stack, "attention_forward", lambda *a: None)
    for name in ("stack_forward", "attention_forward", "shifted_cross_entropy"):
        monkeypatch.setattr(_train, name, lambda *a: None)


def close(got, want, tol):
    return ((got.float() - want.float()).norm() / want.float().norm().clamp_min(1e-12)).item() <= tol


def step(model, ids):
    model.zero_grad(set_to_none=True)
    with torch.enable_grad():  # (other tests may have turned it off)
        out = model(ids, labels=ids)
        out["loss"].backward()
    return out, {n: p.grad for n, p in model.named_parameters()}


@pytest.mark.parametrize("place", ["layers.0.attention", "layers.0.attention.qkv_proj", "layers.1.mlp", "layers.1.mlp.fc2",
                                   "layers.0.norm_mlp", "norm", "lm_head", "embed_tokens"])
@pytest.mark.parametrize("pre", [False, True])
def test_backward_hooks_of_submodules_fire(place, pre):
    model, ids = make()
    mod, seen = model.get_submodule(place), []
    # (the residual add and the norm behind it are one call of add_forward: module by module norm_mlp is not called either)
    register = mod.register_full_backward_pre_hook if pre else mod.register_full_backward_hook
    handle = register(lambda *a: seen.append(1))
    with torch.enable_grad():
        assert _train.stack_forward(model, ids) is None
    step(model, ids)
    assert seen or place in ("layers.0.norm_mlp", "norm")
    handle.remove()
    with torch.enable_grad():
        assert _train.stack_forward(model, ids) is not None


@pytest.mark.parametrize("register", ["register_module_full_backward_hook", "register_module_full_backward_pre_hook"])
def test_global_backward_hooks_fire(register):
    model, ids = make()
    seen = []
    handle = getattr(nn_module, register)(lambda mod, *a: seen.append(type(mod)))
    try:
        step(model, ids)
    finally:
        handle.remove()
    assert nn.Linear in seen


@pytest.mark.parametrize("block_sparse", [False, True])
def test_backward_hook_inside_an_attention_module(block_sparse):
    model, _ = make(block_sparse)
    attn, seen = model.layers[0].attention, []
    attn.out_proj.register_full_backward_hook(lambda *a: seen.append(1))
    with torch.enable_grad():
        x = torch.randn(2, 40, 128, device=DEV, dtype=BF16, requires_grad=True)
        attn(x).sum().backward()
    assert seen == [1]


@pytest.mark.parametrize("block_sparse", [False, True])
def test_forward_hook_of_the_modules_dropout(block_sparse):
    """(an Identity where the rate is 0; the one call skips it)"""
    attn, seen = make(block_sparse)[0].layers[0].attention, []
    attn.dropout.register_forward_hook(lambda *a: seen.append(1))
    with torch.no_grad():
        attn(torch.randn(2, 40, 128, device=DEV, dtype=BF16))
    assert seen == [1]


@pytest.mark.parametrize("place", ["layers.0.attention", "layers.1.mlp", "layers.0.attention.out_proj"])
@pytest.mark.parametrize("train", [False, True])
def test_a_forward_replaced_on_the_instance_is_called(place, train):
    model, ids = make()
    mod, seen = model.get_submodule(place), []
    own = mod.forward
    mod.forward = lambda *a, **k: (seen.append(1), own(*a, **k))[1]
    if train:
        step(model, ids)
    else:
        with torch.no_grad():
            model(ids)
    assert seen


def _window(m):
    m.layers[1].attention.window_size = 3


def _eps(m):
    m.layers[1].norm_mlp.eps = 0.5


def _append(m):
    m.layers.append(make(layers=1, seed=5)[0].layers[0])


def _bias(m):
    m.layers[0].attention.qkv_proj.bias = nn.Parameter(torch.full((384,), 0.5, device=DEV, dtype=BF16))


def _head_bias(m):
    m.lm_head.bias = nn.Parameter(torch.linspace(-1, 1, 128, device=DEV, dtype=BF16))


def _transposed(m):
    w = m.layers[0].attention.out_proj.weight
    w.data = w.data.t()


def _retyped(m):
    for p in m.parameters():
        p.data = (p.data.float() * 0.25).to(torch.float16).view(BF16).view(torch.float16)


def _max_norm(m):
    m.embed_tokens.max_norm = 0.05


@pytest.mark.parametrize("change", [_window, _eps, _append, _bias, _head_bias, _transposed, _retyped, _max_norm],
                         ids=lambda f: f.__name__[1:])
def test_the_model_as_it_is_at_the_call(change, monkeypatch):
    """Changed between two calls: the second gives what a model that never had a first call gives."""
    model, ids = make(tie_weights=False)
    model.eval()
    with torch.no_grad():
        first = model(ids)["logits"]
        change(model)
        got = model(ids)["logits"]
        module_by_module(monkeypatch)
        want = model(ids)["logits"]
    _native.poll_status(torch.device(DEV))
    assert not torch.equal(first, got)
    assert got.dtype == want.dtype and close(got, want, 2e-2)
    assert not close(first.to(want.dtype), want, 2e-2)  # (the change is large enough to be told from rounding)


def _shared_mlp(m):
    m.layers[1].mlp.fc1.weight = m.layers[0].mlp.fc1.weight


def _shared_block(m):
    m.layers[1] = m.layers[0]


def _shared_norm(m):
    m.layers[0].norm_mlp = m.layers[0].norm_attn


@pytest.mark.parametrize("share", [_shared_mlp, _shared_block, _shared_norm], ids=lambda f: f.__name__[1:])
def test_gradients_of_shared_parameters_add_up(share, monkeypatch):
    model, ids = make()
    share(model)
    _, got = step(model, ids)
    module_by_module(monkeypatch)
    _, want = step(model, ids)
    for name in want:
        assert close(got[name], want[name], 6e-2), name


@pytest.mark.parametrize("n_p", [0, 3])
def test_the_loss_depends_on_the_logits_that_are_returned(n_p):
    """Their gradient is there to be kept, hooked and added to."""
    model, ids = make(n_p=n_p)
    with torch.enable_grad():
        out = model(ids, labels=ids)
        logits = out["logits"]
        logits.retain_grad()
        out["loss"].backward()
        a = logits.detach().float().requires_grad_(True)
        torch.nn.functional.cross_entropy(a[:, :-1].reshape(-1, 128), ids[:, 1:].reshape(-1)).backward()
        assert close(logits.grad, a.grad, 1e-2)

        def grads(two_terms, factor):
            model.zero_grad(set_to_none=True)
            out = model(ids, labels=ids)
            if factor != 1:
                out["logits"].register_hook(lambda g: g * factor)
            total = out["loss"] + (out["logits"].float().square().mean() if two_terms else 0.0)
            total.backward()
            return {n: p.grad.clone() for n, p in model.named_parameters()}

        one, doubled = grads(False, 1), grads(False, 2)
        for name in one:
            assert close(doubled[name], 2 * one[name].float(), 3e-2), name
        both = grads(True, 1)
        model.zero_grad(set_to_none=True)
        model(ids)["logits"].float().square().mean().backward()
        for name, prm in model.named_parameters():
            assert close(both[name], one[name].float() + prm.grad.float(), 3e-2), name


def test_a_gradient_of_the_logits_at_an_odd_address():
    model, ids = make(n_p=0)
    with torch.enable_grad():
        logits = model(ids)["logits"]
        extra = torch.zeros(3, device=DEV, dtype=BF16, requires_grad=True)
        g = torch.randn(3 + logits.numel(), device=DEV, dtype=BF16)
        torch.cat([extra, logits.reshape(-1)]).backward(g)  # the second part of g: contiguous, 6 bytes into it
        got = {n: p.grad.clone() for n, p in model.named_parameters()}
        model.zero_grad(set_to_none=True)
        model(ids)["logits"].backward(g[3:].clone().view_as(logits))
    for name, prm in model.named_parameters():
        assert close(got[name], prm.grad, 1e-2), name


def test_options_of_the_embedding_tables(monkeypatch):
    model, ids = make(tie_weights=False)
    step(model, ids)
    model.embed_tokens.padding_idx = int(ids[0, 0])
    _, got = step(model, ids)
    assert not got["embed_tokens.weight"][ids[0, 0]].any()
    model.embed_tokens.padding_idx = None
    model.embed_tokens.scale_grad_by_freq = True
    _, got = step(model, ids)
    module_by_module(monkeypatch)
    _, want = step(model, ids)
    assert close(got["embed_tokens.weight"], want["embed_tokens.weight"], 5e-2)


def test_deterministic_algorithms_when_asked_for():
    """Tokens that repeat a thousand times: sums in no fixed order would differ between the passes."""
    model, _ = make(vocab=64)
    g = torch.Generator(device=DEV).manual_seed(1)
    ids = torch.randint(0, 4, (300, 60), generator=g, device=DEV)
    torch.use_deterministic_algorithms(True, warn_only=True)
    try:
        with torch.enable_grad():
            assert _train.stack_forward(model, ids) is None
        grads = [step(model, ids)[1]["embed_tokens.weight"].clone() for _ in range(4)]
    finally:
        torch.use_deterministic_algorithms(False)
    for g2 in grads[1:]:
        assert torch.equal(grads[0], g2)


class _Scaled(TitanMAC):
    def _embed(self, input_ids, first_position=0):
        return super()._embed(input_ids, first_position) * 3


class _Counting(TitanMAC):
    def decode_step(self, *a):
        self.steps = getattr(self, "steps", 0) + 1
        return super().decode_step(*a)


class _Swapped(WindowedAttention):
    def split_qkv(self, qkv):
        q, k, v = super().split_qkv(qkv)
        return k, q, v


class _Halved(BlockSparseAttention):
    def stacked_conv_weight(self):
        return super().stacked_conv_weight() / 2


def test_a_subclass_that_embeds_otherwise(monkeypatch):
    model, ids = make()
    model.__class__ = _Scaled
    plain, _ = make()
    _, got = step(model, ids)
    with torch.no_grad():
        fwd, pre = model(ids)["logits"], model.prefill(ids)[0]
        assert not close(fwd, plain(ids)["logits"], 5e-2)
        module_by_module(monkeypatch)
        assert close(fwd, model(ids)["logits"], 2e-2) and close(pre, model.prefill(ids)[0], 2e-2)
    _, want = step(model, ids)
    for name in want:
        assert close(got[name], want[name], 6e-2), name


@pytest.mark.parametrize("on_the_instance", [False, True])
def test_generate_takes_the_steps_of_a_subclass(on_the_instance):
    model, ids = make()
    want = model.generate(ids, 5)
    if on_the_instance:
        own, model.steps = model.decode_step, 0

        def counted(*a):
            model.steps += 1
            return own(*a)

        model.decode_step = counted
    else:
        model.__class__ = _Counting
    got = model.generate(ids, 5, use_cuda_graph=False)
    assert model.steps == 4 and torch.equal(got, want)


def test_attention_modules_with_parts_of_their_own():
    with torch.device(DEV):
        win = WindowedAttention(WindowConfig(window_size=16, num_heads=2, head_dim=64, n_persistent=3)).to(BF16)
        sparse = BlockSparseAttention(128, 2, window_size=32, n_persistent=3).to(BF16)
        x = torch.randn(2, 40, 128, device=DEV).to(BF16)
    for mod, sub, train in ((win, _Swapped, False), (sparse, _Halved, False), (sparse, _Halved, True)):
        with torch.set_grad_enabled(train):
            base = mod(x)
            mod.__class__ = sub
            own = mod(x)
            mod.__class__ = sub.__bases__[0]
        assert not close(own, base, 5e-2)


def test_another_kind_of_embedding():
    model, ids = make(tie_weights=False)
    model.eval()
    with torch.no_grad():
        want, cont = model(ids)["logits"], model.generate(ids, 4)
        model.embed_tokens = nn.Sequential(model.embed_tokens)  # has no weight of its own
        assert close(model(ids)["logits"], want, 2e-2)
        assert torch.equal(model.generate(ids, 4)[:, :30], cont[:, :30])
    step(model, ids)
    assert model.embed_tokens[0].weight.grad is not None


def test_tables_of_another_type_than_the_layers():
    """A 16-bit token table in an fp32 model: the embedded rows, and so the keys in the caches, are fp32."""
    model, ids = make(tie_weights=False)
    model = model.float().eval()
    pos = torch.full((2,), 30, dtype=torch.int32, device=DEV)

    def run():
        logits, caches = model.prefill(ids)
        assert caches[0].dtype == torch.float32
        return logits, model.decode_step(ids[:, 0], pos, caches)

    want = run()  # (the table's values are 16-bit ones: the model came from bf16)
    model.embed_tokens.to(BF16)
    got = run()
    for a, b in zip(got, want):
        assert close(a, b, 1e-5)

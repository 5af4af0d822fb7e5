"""Host-side behaviour of the drop-in module that needs no GPU: construction, state_dict
compatibility and the exceptions the reference raises in the same situations."""

import pytest
import torch

from titanmac_b200 import BlockSparseAttention, TitanMACConfig, WindowConfig, WindowedAttention, _native, _stack


def test_constructor_accepts_both_config_kinds():
    a = WindowedAttention(WindowConfig(window_size=8, num_heads=4, head_dim=16, n_persistent=2))
    assert (a.d_model, a.n_heads, a.d_head, a.window_size, a.num_persistent, a.causal, a.dropout_p) == (
        64, 4, 16, 8, 2, True, 0.0)
    b = WindowedAttention(TitanMACConfig(d_model=640, n_heads=10, window_size=512, n_persistent=16))
    assert (b.d_model, b.n_heads, b.d_head, b.window_size, b.num_persistent) == (640, 10, 64, 512, 16)
    assert isinstance(b.dropout, torch.nn.Identity)


def test_state_dict_keys_and_shapes_match_the_reference_module():
    m = WindowedAttention(TitanMACConfig(d_model=128, n_heads=2))
    sd = m.state_dict()
    assert list(sd) == ["qkv_proj.weight", "out_proj.weight"]
    assert sd["qkv_proj.weight"].shape == (384, 128) and sd["out_proj.weight"].shape == (128, 128)


def test_config_errors():
    with pytest.raises(ValueError):
        TitanMACConfig(d_model=641, n_heads=10).d_head
    with pytest.raises(ValueError):
        TitanMACConfig(d_model=641, n_heads=10).validate()
    with pytest.raises(ValueError):
        TitanMACConfig(n_persistent=5000).validate()
    with pytest.raises(ValueError):
        TitanMACConfig(window_size=-1).validate()
    TitanMACConfig().validate()

    class Odd:  # d_model that is not heads * d_head trips the module's own assertion
        d_model, n_heads, d_head, window_size, n_persistent, causal, attention_dropout = 100, 3, 32, 4, 1, True, 0.0

    with pytest.raises(AssertionError):
        WindowedAttention(Odd())


def test_forward_raises_like_the_reference_before_any_device_work():
    m = WindowedAttention(WindowConfig(window_size=4, num_heads=2, head_dim=8, n_persistent=16)).eval()
    for L in (1, 16):  # n_persistent >= length
        with pytest.raises(ValueError, match="must be < seq_len"):
            m(torch.zeros(1, L, 16))
    neg = WindowedAttention(WindowConfig(window_size=-1, num_heads=2, head_dim=8, n_persistent=1)).eval()
    with pytest.raises(ValueError, match="non-negative"):
        neg(torch.zeros(1, 8, 16))


def test_unsupported_modes_and_missing_device_fail_loudly():
    m = WindowedAttention(WindowConfig(window_size=4, num_heads=2, head_dim=8, n_persistent=1)).eval()
    x = torch.zeros(1, 8, 16)
    with pytest.raises(NotImplementedError):
        m(x, attn_mask=torch.ones(8, 8, dtype=torch.bool))
    with pytest.raises(RuntimeError, match="no CPU path"):
        m(x)
    nc = WindowedAttention(WindowConfig(window_size=4, num_heads=2, head_dim=8, n_persistent=1, causal=False))
    with pytest.raises(NotImplementedError):
        nc(x)
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        _native.prefill(torch.zeros(1, 1, 8, 8), torch.zeros(1, 1, 8, 8), torch.zeros(1, 1, 8, 8), 4, 1)


@pytest.mark.parametrize("sparse", [False, True])
def test_one_call_plan_only_for_inputs_and_weights_of_the_modules_own_shapes(sparse):
    """The library takes its extents from the module: anything narrower would be read and written out of bounds."""
    def module():
        m = BlockSparseAttention(d_model=640, n_heads=10) if sparse else WindowedAttention(TitanMACConfig(d_model=640, n_heads=10))
        return m.to(torch.bfloat16)

    def plan(m, width=640):
        x = torch.zeros(2, 24, width, dtype=torch.bfloat16)
        return _stack.attention_plan(m, x, 0, 64 if sparse else 0, 0.125)

    bf16 = dict(bias=False, dtype=torch.bfloat16)
    assert plan(module()) is not None
    for width in (8, 128, 632, 648, 1280):
        assert plan(module(), width) is None
    for name, shape in (("qkv_proj", (640, 640)), ("qkv_proj", (640, 1920 - 64)), ("qkv_proj", (640, 1920 + 64)), ("qkv_proj", (128, 1920)),
                        ("out_proj", (640, 128)), ("out_proj", (640, 648)), ("out_proj", (128, 640))):
        m = module()
        setattr(m, name, torch.nn.Linear(*shape, **bf16))
        assert plan(m) is None, (name, shape)
    for name in ("qkv_proj", "out_proj"):
        m = module()
        getattr(m, name).to("meta")  # (another device than the input's)
        assert plan(m) is None, name
    for name in ("qkv_proj", "out_proj"):
        m = module()
        lin = getattr(m, name)
        w = lin.weight.detach()
        del lin.weight
        lin.weight = w  # a plain tensor, as wrappers that flatten parameters leave it
        assert plan(m) is None, name
    m = module()
    m.n_heads = 20
    assert plan(m) is None
    if sparse:
        for conv in (torch.nn.Conv1d(64, 64, 4, groups=64, **bf16), torch.nn.Conv1d(640, 640, 3, groups=640, **bf16)):
            m = module()
            m.conv_k = conv
            assert plan(m) is None
        m = module()
        m.conv_v.to("meta")
        assert plan(m) is None

"""The training step as two library calls (``tmw_stack_train_*``, ``tmw_cross_entropy``) and the one-call forwards against the
same computation module by module."""

import ctypes

import pytest
import torch

from titanmac_b200 import TitanMAC, TitanMACConfig, _native, _stack, _train

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def make(dtype, heads, dh, window, Np, vocab, block_sparse, layers=2, seed=0):
    D = heads * dh
    cfg = TitanMACConfig(vocab_size=vocab, d_model=D, n_heads=heads, n_layers=layers, d_ff=2 * D + 96, max_seq_len=1024,
                         window_size=window, n_persistent=Np, use_block_sparse=block_sparse, block_size=32)
    g = torch.Generator(device=DEV).manual_seed(seed)
    with torch.device(DEV):
        model = TitanMAC(cfg)
    with torch.no_grad():
        for name, prm in model.named_parameters():
            prm.normal_(1.0 if name.endswith("scale") else 0.0, 0.1 if name.endswith(("scale", "bias")) else 0.04, generator=g)
    return model.to(dtype), g


def module_by_module(monkeypatch):
    monkeypatch.setattr(_stack, "table_of", lambda m: None)
    monkeypatch.setattr(_stack, "attention_forward", lambda *a: None)
    for name in ("stack_forward", "attention_forward", "shifted_cross_entropy"):
        monkeypatch.setattr(_train, name, lambda *a: None)


def close(got, want, tol):
    return ((got.float() - want.float()).norm() / want.float().norm().clamp_min(1e-12)).item() <= tol


@pytest.mark.parametrize("B,T,dtype,heads,dh,window,Np,vocab,block_sparse", [
    (1, 1, torch.bfloat16, 2, 64, 8, 3, 512, False),      # one token: no label is left
    (2, 61, torch.bfloat16, 2, 64, 16, 16, 1000, False),  # 154 rows: two row tiles, a ragged last one
    (3, 130, torch.float16, 3, 64, 32, 5, 776, True),     # odd widths (192), the convolutions' strips cut short
    (2, 200, torch.bfloat16, 1, 128, 40, 0, 4096, False), # no persistent rows
    (8, 1001, torch.bfloat16, 4, 64, 64, 8, 640, True),   # k = 8072 rows in the weights' gradients: cut into ranges
    (4, 1024, torch.float16, 5, 128, 100, 16, 2048, False),  # d_model 640: column tiles narrower than 256
    (5, 1000, torch.bfloat16, 8, 64, 40, 8, 512, False),     # norms of 512 columns, three rows to a warp
    (5, 1000, torch.bfloat16, 8, 128, 40, 8, 512, False),    # 1024 columns
    (5, 1000, torch.float16, 14, 64, 40, 8, 512, False),     # 896
    (2, 150, torch.float16, 16, 128, 40, 4, 512, False),     # 2048 columns, the widest
])
def test_training_step_equals_module_by_module(B, T, dtype, heads, dh, window, Np, vocab, block_sparse, monkeypatch):
    model, g = make(dtype, heads, dh, window, Np, vocab, block_sparse)
    ids = torch.randint(0, vocab, (B, T), generator=g, device=DEV)
    labels = torch.randint(0, vocab, (B, T), generator=g, device=DEV)
    labels[torch.rand(B, T, generator=g, device=DEV) < 0.2] = -100  # ignored
    scale = 1.0 if dtype == torch.bfloat16 else 64.0

    def step():
        model.zero_grad(set_to_none=True)
        with torch.enable_grad():  # (other tests may have turned it off)
            out = model(ids, labels=labels)
            if T > 1:
                (out["loss"] * scale).backward()
        return out["loss"].detach(), out["logits"].detach(), {n: p.grad for n, p in model.named_parameters()}

    loss, logits, grads = step()
    _native.poll_status(torch.device(DEV))
    module_by_module(monkeypatch)
    want_loss, want_logits, want = step()
    tol = 3e-2 if dtype == torch.bfloat16 else 6e-3
    assert close(logits, want_logits, tol)
    if T == 1:
        return
    assert abs(loss.item() - want_loss.item()) <= tol * abs(want_loss.item())
    for name, ref in want.items():
        assert (grads[name] is None) == (ref is None), name
        if ref is not None:
            assert grads[name].dtype == dtype and close(grads[name], ref, 2 * tol), name


@pytest.mark.parametrize("B,T,dtype,heads,dh,Np,block_sparse", [
    (1, 1, torch.bfloat16, 2, 64, 1, False), (2, 33, torch.float16, 3, 64, 0, False), (1, 400, torch.bfloat16, 1, 128, 17, True),
    (3, 127, torch.bfloat16, 4, 64, 16, True),
])
def test_forward_equals_module_by_module(B, T, dtype, heads, dh, Np, block_sparse, monkeypatch):
    model, g = make(dtype, heads, dh, 48, Np, 520, block_sparse)
    model.eval()
    ids = torch.randint(0, 520, (B, T), generator=g, device=DEV)
    x = torch.randn(B, T + max(Np, 1), heads * dh, generator=g, device=DEV).to(dtype)
    attn = model.layers[0].attention
    with torch.no_grad():
        got = model(ids)["logits"], attn(x)
        _native.poll_status(torch.device(DEV))
        module_by_module(monkeypatch)
        want = model(ids)["logits"], attn(x)
    tol = 2e-2 if dtype == torch.bfloat16 else 4e-3
    assert close(got[0], want[0], tol) and close(got[1], want[1], tol)


@pytest.mark.parametrize("block_sparse", [False, True])
@pytest.mark.parametrize("wanted", [("x",), ("qkv_proj",), ("out_proj",), ("x", "out_proj"), ("qkv_proj", "out_proj"), ("conv_k",),
                                    ("x", "conv_q", "conv_v")])
def test_only_the_gradients_that_are_wanted(block_sparse, wanted, monkeypatch):
    """The attention module's backward asks the library for these alone, and they are what they are with all the others."""
    if not block_sparse and any(n.startswith("conv") for n in wanted):
        pytest.skip("no convolutions")
    model, g = make(torch.bfloat16, 2, 64, 40, 5, 64, block_sparse, layers=1)
    attn = model.layers[0].attention
    x = torch.randn(3, 700, 128, generator=g, device=DEV).to(torch.bfloat16)
    dy = torch.randn(3, 700, 128, generator=g, device=DEV).to(torch.bfloat16)

    def grads(names):
        out = {"x": x.clone().requires_grad_("x" in names)}
        for name, prm in attn.named_parameters():
            prm.grad = None
            prm.requires_grad_(name.split(".")[0] in names)
        with torch.enable_grad():
            attn(out["x"]).backward(dy)
        _native.poll_status(torch.device(DEV))
        return {"x": out["x"].grad, **{n.split(".")[0]: p.grad for n, p in attn.named_parameters()}}

    want = grads(["x"] + [n.split(".")[0] for n, _ in attn.named_parameters()])
    asked, real = [], _native.lib()

    class Spy:
        def __getattr__(self, name):
            return getattr(real, name)

        def tmw_attention_train_backward(self, *a):
            asked.append({n for n, p in [("x", a[9])] + [(n, getattr(a[10]._obj, n)) for n, _ in a[10]._obj._fields_] if p})
            return real.tmw_attention_train_backward(*a)

    monkeypatch.setattr(_native, "lib", lambda: Spy())
    got = grads(wanted)
    assert asked == [{n.replace("qkv_proj", "w_qkv").replace("out_proj", "w_out") for n in wanted}]
    for name in want:
        assert (got[name] is None) == (name not in wanted)
        # (a filter's gradient is added up with atomics: the order of its fp32 sums is not fixed)
        assert name not in wanted or (close(got[name], want[name], 1e-2) if "conv" in name else torch.equal(got[name], want[name])), name


@pytest.mark.parametrize("rows,taps", [(6000, 0), (6001, 4)])
def test_scratch_aligned_to_16_bytes(rows, taps):
    """Scratch and saved activations need 16 bytes of alignment, no more: the weights' gradients (k = rows, cut into ranges whose fp32
    sums lie in the scratch) are bit for bit what they are with scratch on a 256-byte boundary, and nothing beyond it is touched."""
    lib, D = _native.lib(), 128
    g = torch.Generator(device=DEV).manual_seed(rows)
    desc = _native.AttentionDesc(_native.TMW_BF16, 1, rows, 2, 64, 40, 5, 32 if taps else 0, taps, 0.0)
    x, dy = (torch.randn(rows, D, generator=g, device=DEV).to(torch.bfloat16) for _ in range(2))
    w_qkv, w_out = ((torch.randn(n, D, generator=g, device=DEV) * 0.1).to(torch.bfloat16) for n in (3 * D, D))
    conv = [(torch.randn(D, taps, generator=g, device=DEV) * 0.5).to(torch.bfloat16) for _ in range(3 if taps else 0)]
    convs = [c.data_ptr() for c in conv] or [None] * 3
    ref, stream = ctypes.byref(desc), _native._stream_ptr(torch.device(DEV))
    n_saved, n_scratch = lib.tmw_attention_train_saved(ref), lib.tmw_attention_train_scratch(ref)

    def run(shift):
        room = torch.full((n_scratch + 512,), 77, dtype=torch.uint8, device=DEV)
        saved = torch.empty(n_saved + 512, dtype=torch.uint8, device=DEV)
        y, dx = torch.empty_like(x), torch.empty_like(x)
        out = [torch.empty_like(w) for w in (w_qkv, w_out)]
        grads = _native.BlockGrads(w_qkv=out[0].data_ptr(), w_out=out[1].data_ptr())
        _native.check(lib.tmw_attention_train_forward(ref, x.data_ptr(), w_qkv.data_ptr(), *convs, w_out.data_ptr(), y.data_ptr(),
                                                      saved.data_ptr() + shift, n_saved, stream))
        _native.check(lib.tmw_attention_train_backward(ref, x.data_ptr(), w_qkv.data_ptr(), *convs, w_out.data_ptr(), dy.data_ptr(),
                                                       saved.data_ptr() + shift, dx.data_ptr(), ctypes.byref(grads),
                                                       room.data_ptr() + shift, n_scratch, stream))
        _native.poll_status(torch.device(DEV))
        assert (room[:shift] == 77).all() and (room[shift + n_scratch:] == 77).all()
        return y, dx, *out

    for got, want in zip(run(16), run(0)):
        assert torch.equal(got, want)


@pytest.mark.parametrize("B,T,d_ff", [
    (1, 40, 256),        # 5 partial rows of the norms, 1 of fc1's bias: one chain each
    (1, 1023, 4096), (1, 1023, 4104),  # 128 partial rows; 16 strips of fc1's bias
    (2, 604, 4096), (2, 604, 4104),    # 151; 19 strips, either side of the columns that share out the threads differently
    (8, 1024, 128),      # 296; weight gradients cut into more than 16 ranges
])
def test_sums_of_partial_results(B, T, d_ff):
    """Every row of the batch is the same token at the same (zero) position, so each sum over the rows is their number times the
    gradient of one row: a part that is missing or counted twice shows.  Tolerance: a part is at least 1/296 of a sum; one rounding
    to fp16 of each of a gradient's factors, on average over the elements, is below 2^-11."""
    heads, vocab = 2, 64
    cfg = TitanMACConfig(vocab_size=vocab, d_model=64 * heads, n_heads=heads, n_layers=1, d_ff=d_ff, max_seq_len=1024, window_size=16,
                         n_persistent=0, use_block_sparse=False)
    g = torch.Generator(device=DEV).manual_seed(d_ff)
    with torch.device(DEV):
        model = TitanMAC(cfg)
    with torch.no_grad():
        for name, prm in model.named_parameters():
            prm.normal_(1.0 if name.endswith("scale") else 0.0, 0.1 if name.endswith(("scale", "bias")) else 0.04, generator=g)
            if "pos" in name:
                prm.zero_()
    model = model.half()
    d_row = torch.randn(vocab, generator=g, device=DEV)

    def grads(B, T, scale):
        model.zero_grad(set_to_none=True)
        with torch.enable_grad():
            logits = model(torch.full((B, T), 7, device=DEV))["logits"]
        assert "_StackTrain" in type(logits.grad_fn).__name__
        logits.backward((d_row * scale).half().expand(B, T, vocab))
        _native.poll_status(torch.device(DEV))
        return {n: p.grad.float() / scale for n, p in model.named_parameters()}

    one, many = grads(1, 1, 1.0), grads(B, T, 2.0 ** -4)
    checked = [n for n in one if "embed" not in n and "attention" not in n and "norm_attn" not in n]
    assert len(checked) >= 5
    for name in checked:
        want = one[name] * (B * T)
        if want.norm() > 0:
            assert ((many[name] - want).norm() / want.norm()).item() <= 2 ** -10, name


@pytest.mark.parametrize("B,T,dtype,heads,dh,d_ff,vocab", [
    (2, 61, torch.bfloat16, 2, 64, 264, 520),       # hidden rows and logits of 16 n + 8 values
    (4, 1024, torch.float16, 2, 128, 2568, 1000),   # more rows, tiles of 256
])
def test_training_step_of_rows_off_the_sectors(B, T, dtype, heads, dh, d_ff, vocab, monkeypatch):
    """The epilogues of such rows (kept GELU argument, its derivative) against the same computation module by module; tolerances as
    above."""
    D = heads * dh
    cfg = TitanMACConfig(vocab_size=vocab, d_model=D, n_heads=heads, n_layers=2, d_ff=d_ff, max_seq_len=1024, window_size=32,
                         n_persistent=5, use_block_sparse=False)
    g = torch.Generator(device=DEV).manual_seed(d_ff)
    with torch.device(DEV):
        model = TitanMAC(cfg)
    with torch.no_grad():
        for name, prm in model.named_parameters():
            prm.normal_(1.0 if name.endswith("scale") else 0.0, 0.1 if name.endswith(("scale", "bias")) else 0.04, generator=g)
    model = model.to(dtype)
    ids = torch.randint(0, vocab, (B, T), generator=g, device=DEV)
    scale = 1.0 if dtype == torch.bfloat16 else 64.0

    def step():
        model.zero_grad(set_to_none=True)
        with torch.enable_grad():
            out = model(ids, labels=ids)
            (out["loss"] * scale).backward()
        _native.poll_status(torch.device(DEV))
        return out["logits"].detach(), {n: p.grad for n, p in model.named_parameters()}

    logits, grads = step()
    module_by_module(monkeypatch)
    want_logits, want = step()
    tol = 3e-2 if dtype == torch.bfloat16 else 6e-3
    assert close(logits, want_logits, tol)
    for name, ref in want.items():
        assert close(grads[name], ref, 2 * tol), name


@pytest.mark.parametrize("shifts", [(16, 0), (0, 16), (16, 16)])
def test_training_step_with_buffers_aligned_to_16_bytes(shifts, monkeypatch):
    """Saved activations and scratch 16 bytes into their allocations, together and one of them alone (an epilogue then reads rows that
    start on sectors and writes rows that do not, or the other way round): bit for bit the gradients of aligned ones."""
    model, g = make(torch.bfloat16, 2, 64, 40, 5, 512, False)
    ids = torch.randperm(512, generator=g, device=DEV)[:450].view(3, 150)  # (each token once: no sum has an order to choose)

    def step(shifts):
        left, empty = list(shifts), torch.empty

        def shifted(*size, **kw):
            if kw.get("dtype") is not torch.uint8:
                return empty(*size, **kw)
            off = left.pop(0)
            return empty(size[0] + 32, **kw)[off:off + size[0]]

        model.zero_grad(set_to_none=True)
        with monkeypatch.context() as m, torch.enable_grad():
            m.setattr(torch, "empty", shifted)
            out = model(ids, labels=ids)
            out["loss"].backward()
            assert not left
        _native.poll_status(torch.device(DEV))
        return out["logits"].detach(), {n: p.grad for n, p in model.named_parameters()}

    want_logits, want = step((0, 0))
    logits, grads = step(shifts)
    assert torch.equal(logits, want_logits)
    for name, ref in want.items():
        assert torch.equal(grads[name], ref), name

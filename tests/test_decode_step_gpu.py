"""The whole decode step as one library call (``tmw_decode_step``) against the same step module by module: every row
count at which the products change their kernel, both head sizes, a vocabulary that is no multiple of eight."""

import pytest
import torch

from titanmac_b200 import TitanMAC, TitanMACConfig, _native, _stack

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def make(dtype, heads, dh, window, Np, vocab, layers=2, seed=0):
    D = heads * dh
    cfg = TitanMACConfig(vocab_size=vocab, d_model=D, n_heads=heads, n_layers=layers, d_ff=3 * D + 32, max_seq_len=256,
                         window_size=window, n_persistent=Np, use_block_sparse=False)
    g = torch.Generator(device=DEV).manual_seed(seed)
    with torch.device(DEV):
        model = TitanMAC(cfg).eval()
    with torch.no_grad():
        for name, prm in model.named_parameters():
            prm.normal_(1.0 if name.endswith("scale") else 0.0, 0.1 if name.endswith(("scale", "bias")) else 0.04, generator=g)
    return model.to(dtype), g


@pytest.mark.parametrize("B,dtype,heads,dh,window,Np,vocab,t", [
    (1, torch.bfloat16, 10, 64, 512, 16, 1003, 200),   # one sequence, a ragged vocabulary
    (8, torch.float16, 4, 128, 70, 0, 5000, 20),       # ring not full yet, no persistent rows
    (16, torch.bfloat16, 2, 64, 33, 5, 512, 100),
    (17, torch.bfloat16, 6, 64, 20, 3, 776, 61),       # the second row tile holds one row
    (32, torch.float16, 3, 128, 64, 16, 333, 64),
    (33, torch.bfloat16, 2, 64, 8, 1, 1000, 0),        # first token; tcgen05 products from here on
    (129, torch.bfloat16, 10, 64, 17, 16, 99, 40),     # two tiles of 128 rows, a ragged vocabulary
    (256, torch.float16, 8, 64, 40, 8, 1024, 41),
])
def test_step_equals_module_by_module(B, dtype, heads, dh, window, Np, vocab, t, monkeypatch):
    model, g = make(dtype, heads, dh, window, Np, vocab)
    ids = torch.randint(0, vocab, (B,), generator=g, device=DEV)
    pos = torch.randint(max(0, t - 3), t + 1, (B,), generator=g, device=DEV, dtype=torch.int32)
    sets = []
    for _ in range(2):
        sets.append(model.new_caches(B, DEV, dtype))
    for a, b in zip(*sets):
        for x, y in zip((a.k_ring, a.v_ring, a.k_pers, a.v_pers), (b.k_ring, b.v_ring, b.k_pers, b.v_pers)):
            x.normal_(0.0, 0.5, generator=g)
            y.copy_(x)
    assert _stack.table_of(model) is not None
    got = model.decode_step(ids, pos, sets[0])
    _native.poll_status(torch.device(DEV))
    monkeypatch.setattr(_stack, "table_of", lambda m: None)
    want = model.decode_step(ids, pos, sets[1])
    tol = 2e-2 if dtype == torch.bfloat16 else 4e-3
    assert got.shape == want.shape == (B, vocab)
    assert ((got.float() - want.float()).norm() / want.float().norm()).item() <= tol
    for a, b in zip(*sets):
        for x, y in ((a.k_ring, b.k_ring), (a.v_ring, b.v_ring)):
            assert ((x.float() - y.float()).norm() / y.float().norm()).item() <= tol


@pytest.mark.parametrize("B,dtype,heads,dh,window,n_p,t", [
    (1, torch.bfloat16, 2, 64, 4094, 3, 200),     # one slot below the rule: the resident kernel
    (3, torch.bfloat16, 2, 128, 2046, 3, 2100),   # one slot below the rule: clusters
    (1, torch.bfloat16, 2, 64, 4095, 3, 0),       # the first token, nothing in the ring
    (3, torch.float16, 4, 64, 4100, 0, 4000),     # ring not full, no persistent rows
    (2, torch.bfloat16, 3, 128, 2047, 16, 9001),  # full
    (24, torch.bfloat16, 2, 64, 5000, 5, 4999),   # 48 pairs; 50 with the next, no longer split on 148 SMs
    (25, torch.bfloat16, 2, 64, 5000, 5, 5000),
    (1, torch.float16, 1, 128, 16384, 1, 30000),
])
def test_long_windows_with_few_pairs(B, dtype, heads, dh, window, n_p, t, monkeypatch):
    """The step's split attention, twice in a row (its counters are left as they were found), against the unsplit kernel."""
    model, g = make(dtype, heads, dh, window, n_p, 128)
    model.embed_positions = torch.nn.Embedding(t + 2, heads * dh, device=DEV, dtype=dtype)
    model.config.max_seq_len = t + 2
    ids = torch.randint(0, 128, (B,), generator=g, device=DEV)
    pos = torch.full((B,), t, dtype=torch.int32, device=DEV)
    pos[0] = max(0, t - 2)
    sets = [model.new_caches(B, DEV, dtype) for _ in range(2)]
    for a, b in zip(*sets):
        b.splits = 0
        for x, y in zip((a.k_ring, a.v_ring, a.k_pers, a.v_pers), (b.k_ring, b.v_ring, b.k_pers, b.v_pers)):
            x.normal_(0.0, 0.5, generator=g)
            y.copy_(x)
    got = [model.decode_step(ids, pos + i, sets[0]) for i in range(2)]
    _native.poll_status(torch.device(DEV))
    monkeypatch.setattr(_stack, "table_of", lambda m: None)
    want = [model.decode_step(ids, pos + i, sets[1]) for i in range(2)]
    tol = 2e-2 if dtype == torch.bfloat16 else 4e-3
    for a, b in zip(got, want):
        assert ((a.float() - b.float()).norm() / b.float().norm()).item() <= tol
    for a, b in zip(*sets):
        for x, y in ((a.k_ring, b.k_ring), (a.v_ring, b.v_ring)):
            assert ((x.float() - y.float()).norm() / y.float().norm()).item() <= tol


@pytest.mark.parametrize("B,heads,one_call", [(2, 32, True), (40, 32, True), (2, 40, False), (40, 40, False)])
def test_widths_around_the_steps_limit(B, heads, one_call, monkeypatch):
    """The step's norms keep a row of at most 4096 in registers: a wider model goes to its modules."""
    model, g = make(torch.bfloat16, heads, 128, 16, 1, 64, layers=1)
    assert _stack.table_of(model).decodes == one_call
    ids = torch.randint(0, 64, (B, 6), generator=g, device=DEV)
    assert model.generate(ids, 3).shape == (B, 9)
    logits, caches = model.prefill(ids)
    pos = torch.full((B,), 6, dtype=torch.int32, device=DEV)
    got = model.decode_step(ids[:, 0], pos, caches)
    _native.poll_status(torch.device(DEV))
    monkeypatch.setattr(_stack, "table_of", lambda m: None)
    want = model.decode_step(ids[:, 0], pos, caches)  # (the step before has written the same keys and values)
    assert ((got.float() - want.float()).norm() / want.float().norm()).item() <= 2e-2


def test_table_follows_the_model():
    """A moved parameter, a replaced module, a hook: the step never uses what the model no longer is."""
    model, g = make(torch.bfloat16, 2, 64, 16, 2, 128)
    caches = model.new_caches(3, DEV, torch.bfloat16)
    ids = torch.tensor([1, 2, 3], device=DEV)
    pos = torch.zeros(3, dtype=torch.int32, device=DEV)
    before = model.decode_step(ids, pos, caches)
    lin = torch.nn.Linear(128, 128, bias=False, device=DEV, dtype=torch.bfloat16)
    model.layers[1].attention.out_proj = lin
    replaced = model.decode_step(ids, pos, caches)
    assert not torch.equal(before, replaced)
    with torch.no_grad():
        lin.weight = torch.nn.Parameter(lin.weight * 2)
    assert not torch.equal(replaced, model.decode_step(ids, pos, caches))
    seen = []
    handle = model.layers[0].mlp.register_forward_hook(lambda *a: seen.append(1))
    model.decode_step(ids, pos, caches)
    handle.remove()
    assert seen == [1] and _stack.table_of(model) is not None


def test_ids_outside_the_table_are_reported():
    model, _ = make(torch.bfloat16, 2, 64, 16, 2, 128)
    caches = model.new_caches(2, DEV, torch.bfloat16)
    model.decode_step(torch.tensor([5, 128], device=DEV), torch.zeros(2, dtype=torch.int32, device=DEV), caches)
    with pytest.raises(_native.TmwError):
        _native.poll_status(torch.device(DEV))
    _native.poll_status(torch.device(DEV))


@pytest.mark.parametrize("B,vocab,new", [(1, 1003, 5), (3, 512, 1), (40, 776, 9), (2, 8, 0)])
def test_generate_equals_argmax_over_steps(B, vocab, new):
    """``tmw_generate`` against a loop of ``decode_step`` and ``argmax``."""
    model, g = make(torch.bfloat16, 2, 64, 20, 3, vocab)
    ids = torch.randint(0, vocab, (B, 11), generator=g, device=DEV)
    got = model.generate(ids, new)
    logits, caches = model.prefill(ids)
    want = [ids]
    pos = torch.full((B,), 11, dtype=torch.int32, device=DEV)
    for _ in range(new):
        want.append(logits.argmax(-1)[:, None])
        logits = model.decode_step(want[-1][:, 0], pos, caches)
        pos += 1
    assert torch.equal(got, torch.cat(want, dim=1))


@pytest.mark.parametrize("B,heads,vocab", [(17, 2, 48000), (64, 2, 20000), (40, 17, 30000), (3, 17, 30000)])
def test_generate_behind_a_wide_head(B, heads, vocab):
    """More than 16 rows or a width above 1024: the head is the tcgen05 product, whose output (megabytes, stored through TMA)
    the choice reads as a dependent launch.  Every token against the ones that steps of their own give."""
    model, g = make(torch.bfloat16, heads, 64, 20, 3, vocab, layers=1)
    for _ in range(3):
        ids = torch.randint(0, vocab, (B, 5), generator=g, device=DEV)
        got = model.generate(ids, 24)
        logits, caches = model.prefill(ids)
        pos = torch.full((B,), 5, dtype=torch.int32, device=DEV)
        for i in range(24):
            token = logits.argmax(-1)
            assert torch.equal(got[:, 5 + i], token), i
            logits = model.decode_step(token, pos, caches)
            pos += 1


def test_greedy_choice_of_ties_and_nan():
    model, _ = make(torch.bfloat16, 2, 64, 20, 0, 5000, layers=1)
    logits = torch.zeros(4, 5000, dtype=torch.bfloat16, device=DEV)
    logits[0, 4321] = logits[0, 17] = 2.0
    logits[1] = -0.0
    logits[1, 600:] = 0.0
    logits[2, 900], logits[2, 100], logits[2, 3] = float("nan"), float("nan"), float("inf")
    logits[3] = -1.0
    logits[3, 4999] = -0.5
    ids = torch.zeros(4, 1, dtype=torch.int64, device=DEV)
    out = _stack.generate(_stack.table_of(model), ids, logits.clone(), model.new_caches(4, DEV, torch.bfloat16), 1)
    assert out[:, 1].tolist() == [17, 0, 100, 4999] == logits.argmax(-1).tolist()

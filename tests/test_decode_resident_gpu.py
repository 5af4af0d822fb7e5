"""The decode step as one resident kernel (up to eight sequences, head_dim 64) against the step module by module and against the
chain of launches that it stands in for: the sizes at which its phases change shape, what must stay in its own sequence,
generation, the step under stream capture and from two threads.  Which kernels ran is read from the profiler."""

import ctypes
import math
import threading

import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from titanmac_b200 import TitanMAC, TitanMACConfig, _native, _stack

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def make(dtype, heads, window, n_p, vocab, layers=2, d_ff=None, positions=256, seed=0):
    D = heads * 64
    cfg = TitanMACConfig(vocab_size=vocab, d_model=D, n_heads=heads, n_layers=layers, d_ff=d_ff or 4 * D, max_seq_len=positions,
                         window_size=window, n_persistent=n_p, use_block_sparse=False)
    g = torch.Generator(device=DEV).manual_seed(seed)
    with torch.device(DEV):
        model = TitanMAC(cfg).eval()
    with torch.no_grad():
        for name, prm in model.named_parameters():
            prm.normal_(1.0 if name.endswith("scale") else 0.0, 0.1 if name.endswith(("scale", "bias")) else 0.04, generator=g)
    return model.to(dtype), g


def filled(model, B, dtype, g, sets=2):
    caches = [model.new_caches(B, DEV, dtype) for _ in range(sets)]
    for group in zip(*caches):
        for tensors in zip(*((c.k_ring, c.v_ring, c.k_pers, c.v_pers) for c in group)):
            tensors[0].normal_(0.0, 0.5, generator=g)
            for t in tensors[1:]:
                t.copy_(tensors[0])
    return caches


def relative(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm()).item()


def is_resident(call):
    """``call()``, and whether the resident kernel ran in it (else the chain did)."""
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as prof:
        out = call()
        torch.cuda.synchronize()
    names = [e.name for e in prof.events()]
    resident, chain = (any(part in n for n in names) for part in ("decode_resident_kernel", "rows_gemm_kernel"))
    assert resident != chain, names
    return out, resident


@pytest.fixture
def take_chain(monkeypatch):
    """Switches the decode calls to the chain of launches: biases that are not aligned to 16 bytes, which the resident kernel
    does not take."""
    kept = []
    arguments = _stack._step_arguments

    def misaligned(table, batch, caches):
        d, blocks, workspace = arguments(table, batch, caches)
        for b, layer in zip(blocks, table.layers_of_test):
            bias = layer.mlp.fc1.bias.detach()
            kept.append(torch.cat([bias.new_zeros(1), bias]))
            b.b_fc1 = ctypes.c_void_p(kept[-1].data_ptr() + bias.element_size())
        return d, blocks, workspace

    def switch(model):
        _stack.table_of(model).layers_of_test = model.layers
        monkeypatch.setattr(_stack, "_step_arguments", misaligned)

    yield switch
    torch.cuda.synchronize()


@pytest.mark.parametrize("B,dtype,heads,window,n_p,vocab,t,layers,d_ff,resident", [
    (1, torch.bfloat16, 1, 0, 0, 7, 0, 1, 32, True),            # the smallest: one key, fewer chunks of k than warps
    (8, torch.float16, 1, 5, 3, 9, 2, 3, 96, True),             # ring not full, fewer keys than warps
    (8, torch.bfloat16, 10, 512, 16, 50000, 600, 2, None, True),  # the default geometry
    (7, torch.float16, 8, 186, 5, 1003, 1000, 2, None, True),   # 16 keys per warp: one tile
    (3, torch.bfloat16, 5, 187, 5, 1000, 300, 2, 1056, True),   # 17: one key in the second; a width that is no multiple of 128
    (2, torch.bfloat16, 10, 751, 16, 512, 800, 2, None, True),  # 64 keys per warp: four tiles, what it holds at once
    (8, torch.float16, 10, 752, 16, 512, 2000, 2, None, True),  # 65: twice
    (1, torch.bfloat16, 2, 4094, 3, 1000, 5000, 2, None, True),  # the longest of few heads: one slot more is split over the chip
    (1, torch.bfloat16, 12, 3000, 1, 520, 3100, 2, 3072, True),  # several times; the widest that it takes
    (4, torch.bfloat16, 13, 40, 2, 512, 60, 2, None, False),    # the next width: the chain
    (8, torch.bfloat16, 2, 40, 2, 512, 60, 2, 3104, False),     # the next hidden width: the chain
    (9, torch.bfloat16, 2, 40, 2, 512, 60, 2, None, False),     # the next number of sequences: the chain
    (2, torch.bfloat16, 1, 20, 2, 512, 30, 33, 64, False),      # the next number of layers: the chain
    (5, torch.bfloat16, 12, 64, 16, 8000, 90, 32, None, True),  # the most layers
])
def test_against_the_modules_and_the_chain(B, dtype, heads, window, n_p, vocab, t, layers, d_ff, resident, monkeypatch, take_chain):
    model, g = make(dtype, heads, window, n_p, vocab, layers, d_ff, positions=t + 4)
    ids = torch.randint(0, vocab, (B,), generator=g, device=DEV)
    pos = torch.randint(max(0, t - 3), t + 1, (B,), generator=g, device=DEV, dtype=torch.int32)
    got_caches, chain_caches, want_caches, before = filled(model, B, dtype, g, sets=4)

    def steps(caches):  # (the second reads what the first has written)
        return [model.decode_step(ids, pos + i, caches) for i in range(2)]

    got, ran = is_resident(lambda: steps(got_caches))
    assert ran == resident
    take_chain(model)
    chain, ran = is_resident(lambda: steps(chain_caches))
    assert not ran
    _native.poll_status(torch.device(DEV))
    monkeypatch.setattr(_stack, "table_of", lambda m: None)
    want = steps(want_caches)
    # rounding to 16 bits through `layers` layers, as between any two kernels of the step
    tol = (2e-2 if dtype == torch.bfloat16 else 4e-3) * max(1.0, (layers / 8) ** 0.5)
    written = torch.zeros((B, window + 1), dtype=torch.bool, device=DEV)
    for i in range(2):
        written[torch.arange(B, device=DEV), (pos.long() + i) % (window + 1)] = True
    for logits, caches in ((got, got_caches), (chain, chain_caches)):
        for a, b in zip(logits, want):
            assert relative(a, b) <= tol, relative(a, b)
        for a, b, old in zip(caches, want_caches, before):
            assert torch.equal(a.k_pers, old.k_pers) and torch.equal(a.v_pers, old.v_pers)
            for ring, other, was in ((a.k_ring, b.k_ring, old.k_ring), (a.v_ring, b.v_ring, old.v_ring)):
                ring, other, was = (r.transpose(1, 2) for r in (ring, other, was))
                assert torch.equal(ring[~written], was[~written])  # nothing but the new rows was written
                assert relative(ring[written], other[written]) <= tol


def test_a_sequence_keeps_its_nan_to_itself():
    """An id outside the table, and a NaN in one sequence's cache, reach that sequence's logits and no others."""
    model, g = make(torch.bfloat16, 4, 40, 3, 256)
    ids = torch.randint(0, 256, (6,), generator=g, device=DEV)
    pos = torch.full((6,), 50, dtype=torch.int32, device=DEV)
    clean, dirty = filled(model, 6, torch.bfloat16, g)
    want = model.decode_step(ids, pos, clean)
    dirty[0].v_ring[4, 1, 7, 9] = float("nan")
    bad = ids.clone()
    bad[2] = 256
    got = model.decode_step(bad, pos, dirty)
    with pytest.raises(_native.TmwError):
        _native.poll_status(torch.device(DEV))
    for b in range(6):
        if b in (2, 4):
            assert torch.isnan(got[b]).all()
        else:
            assert torch.equal(got[b], want[b])


@pytest.mark.parametrize("bad", [2 ** 31 - 1, 2 ** 31 - 2, 256, -1, -2 ** 31])
def test_positions_outside_the_table(bad):
    """Such a sequence's logits are NaN and its new key and value (NaN too) go to the slot of that position
    (of position 0, if negative); the others are as without it."""
    model, g = make(torch.bfloat16, 4, 40, 3, 256)
    ids = torch.randint(0, 256, (3,), generator=g, device=DEV)
    pos = torch.full((3,), 50, dtype=torch.int32, device=DEV)
    clean, dirty = filled(model, 3, torch.bfloat16, g)
    before = [(c.k_ring.clone(), c.v_ring.clone()) for c in dirty]
    want = model.decode_step(ids, pos, clean)
    _native.poll_status(torch.device(DEV))
    pos[1] = bad
    got = model.decode_step(ids, pos, dirty)
    with pytest.raises(_native.TmwError):
        _native.poll_status(torch.device(DEV))
    assert torch.isnan(got[1]).all() and torch.equal(got[0::2], want[0::2])
    slot = max(bad, 0) % 41
    for a, b, (k, v) in zip(dirty, clean, before):
        for ring, other, old in ((a.k_ring, b.k_ring, k), (a.v_ring, b.v_ring, v)):
            assert torch.equal(ring[0::2], other[0::2])
            assert torch.isnan(ring[1, :, slot]).all()
            old[1, :, slot] = ring[1, :, slot]
            assert torch.equal(ring[1].view(torch.int16), old[1].view(torch.int16))


@pytest.mark.parametrize("dtype,scale", [(torch.bfloat16, 2.0 ** -40), (torch.float16, 2.0 ** -9), (torch.bfloat16, 0.3), (torch.float16, 3.0),
                                         (torch.float16, 2.0 ** 13), (torch.bfloat16, 2.0 ** 55)])
@pytest.mark.parametrize("heads", [1, 10])
def test_norm_of_the_head(dtype, scale, heads):
    """Layers that add nothing and a head that is the identity: the logits are the embedded rows, normalised."""
    D = heads * 64
    model, g = make(dtype, heads, 8, 0, D, layers=1)
    with torch.no_grad():
        for lin in (model.layers[0].attention.out_proj, model.layers[0].mlp.fc2):
            for prm in lin.parameters():
                prm.zero_()
        model.embed_positions.weight.zero_()
        model.embed_tokens.weight.normal_(0.0, scale, generator=g)
        model.norm.scale.fill_(1.0)
        model.lm_head.weight = torch.nn.Parameter(torch.eye(D, dtype=dtype, device=DEV))
    ids = torch.arange(8, device=DEV) % D
    got = model.decode_step(ids, torch.zeros(8, dtype=torch.int32, device=DEV), model.new_caches(8, DEV, dtype)).double()
    x = model.embed_tokens.weight[ids].double()
    want = x / torch.sqrt(x.square().mean(-1, keepdim=True) + model.config.norm_eps)
    # one rounding to 16 bits (at most u, or half of fp16's smallest step), in front of it a few of 32 bits
    u, floor = (2.0 ** -8, 0.0) if dtype == torch.bfloat16 else (2.0 ** -11, 2.0 ** -25)
    assert ((got - want).abs() <= (u + 2.0 ** -20) * want.abs() + floor).all()


@pytest.mark.parametrize("chain", [False, True])
@pytest.mark.parametrize("B,dtype,vocab,new", [(1, torch.bfloat16, 1003, 30), (8, torch.float16, 4001, 9), (5, torch.bfloat16, 8, 2)])
def test_generation_equals_steps(B, dtype, vocab, new, chain, take_chain):
    model, g = make(dtype, 6, 20, 3, vocab, layers=3)
    ids = torch.randint(0, vocab, (B, 11), generator=g, device=DEV)
    if chain:
        take_chain(model)
    got, resident = is_resident(lambda: model.generate(ids, new))
    assert resident != chain
    logits, caches = model.prefill(ids)
    pos = torch.full((B,), 11, dtype=torch.int32, device=DEV)
    for i in range(new):
        token = logits.argmax(-1)
        assert torch.equal(got[:, 11 + i], token), i
        logits = model.decode_step(token, pos, caches)
        pos += 1


def test_steps_from_two_threads():
    """Each thread on a stream of its own, with its own caches: what the steps give one after the other."""
    model, g = make(torch.bfloat16, 10, 100, 3, 3000, layers=4)
    ids = torch.randint(0, 3000, (2, 4), generator=g, device=DEV)
    pos = torch.full((4,), 150, dtype=torch.int32, device=DEV)
    alone, together = filled(model, 4, torch.bfloat16, g), [model.new_caches(4, DEV, torch.bfloat16) for _ in range(2)]
    for a, b in zip(alone, together):
        for x, y in zip(a, b):
            for name in ("k_ring", "v_ring", "k_pers", "v_pers"):
                getattr(y, name).copy_(getattr(x, name))
    positions = [pos + i for i in range(40)]
    want = [[model.decode_step(ids[k], p, alone[k]) for p in positions] for k in range(2)]
    torch.cuda.synchronize()
    got, streams = [None, None], [torch.cuda.Stream(DEV) for _ in range(2)]

    def work(k):
        with torch.cuda.stream(streams[k]):
            got[k] = [model.decode_step(ids[k], p, together[k]) for p in positions]

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    torch.cuda.synchronize()
    _native.poll_status(torch.device(DEV))
    for k in range(2):
        assert all(torch.equal(a, b) for a, b in zip(got[k], want[k]))


def test_step_under_capture():
    model, g = make(torch.bfloat16, 4, 30, 2, 256)
    ids = torch.randint(0, 256, (3,), generator=g, device=DEV)
    pos = torch.full((3,), 40, dtype=torch.int32, device=DEV)
    eager, captured = filled(model, 3, torch.bfloat16, g)
    want = [model.decode_step(ids, pos + i, eager) for i in range(3)]
    graph = torch.cuda.CUDAGraph()
    static = pos.clone()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        logits = model.decode_step(ids, static, captured)
    for i in range(3):
        graph.replay()
        assert torch.equal(logits, want[i]), i
        static += 1


def one_head(dtype, window, query):
    """A model of one layer and one head whose query is ``query`` e_0, whose new key and value are zeros and whose logits are the
    normalised row 64 e_0 + attention; and its cache of zeros."""
    D = 64
    cfg = TitanMACConfig(vocab_size=D, d_model=D, n_heads=1, n_layers=1, d_ff=4 * D, max_seq_len=2 * window, window_size=window,
                         n_persistent=0, use_block_sparse=False)
    with torch.device(DEV):
        model = TitanMAC(cfg).eval().to(dtype)
    with torch.no_grad():
        for name, prm in model.named_parameters():
            prm.fill_(1.0 if name.endswith("scale") else 0.0)
        model.embed_tokens.weight[:, 0] = 64.0  # whose norm is 8 e_0
        attn = model.layers[0].attention
        attn.qkv_proj.weight[0, 0] = query / 8
        attn.out_proj.weight.copy_(torch.eye(D))
        model.lm_head.weight = torch.nn.Parameter(torch.eye(D, dtype=dtype, device=DEV))
    caches = model.new_caches(1, DEV, dtype)
    caches[0].k_ring.zero_()
    caches[0].v_ring.zero_()
    return model, caches


def check_row(model, caches, t, row):
    """The step's logits against those of the attention's output ``row`` (64 bits, first element zero)."""
    row = row + 64.0 * torch.nn.functional.one_hot(torch.tensor(0, device=DEV), 64)
    want = row / torch.sqrt(row.square().mean() + model.config.norm_eps)
    got = model.decode_step(torch.tensor([3], device=DEV), torch.tensor([t], dtype=torch.int32, device=DEV), caches)[0].double()
    # Roundings to 16 bits, u each, of the attention's output, the normalised row and the logit (the query and all sums with one
    # nonzero term are exact), and one u for the rest; in fp16 each of them may lie below 2^-14, where the spacing is 2^-24
    fp16 = caches[0].dtype == torch.float16
    u = 2.0 ** (-11 if fp16 else -8)
    floor = 2.0 ** -25 * (want[1:].abs() / row[1:].abs() + 2) if fp16 else 0.0
    assert ((got[1:] - want[1:]).abs() <= 4 * u * want[1:].abs() + floor).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("window,exponent", [(300, -12.6), (300, -18.6), (300, -23.4), (1500, -23.4), (300, -31.3)])
def test_small_weights_with_large_values(dtype, window, exponent):
    """Every eighth key has score 0 and value 0, the others weigh 2^exponent and carry large values: the output is nothing but
    small weights, each of which counts with the precision of fp32 (a 16-bit part of its own has none left of them in fp16)."""
    model, caches = one_head(dtype, window, 8.0)
    k, v = caches[0].k_ring, caches[0].v_ring
    small = torch.arange(window + 1, device=DEV) % 8 != 0
    k[0, 0, :, 0] = small * exponent * math.log(2.0)  # q k / sqrt(64) = k[0]
    top = 6e4 if dtype == torch.float16 else 2.0 ** 40  # (bf16: so that the smallest weights matter there too)
    v.uniform_(0.25, 1.0, generator=torch.Generator(device=DEV).manual_seed(1)).mul_(top).mul_(small[:, None])
    v[..., 0] = 0.0
    t = 2 * window - 3
    weight, values = torch.exp(k[0, 0, :, 0].double()), v[0, 0].double()
    weight[t % (window + 1)], values[t % (window + 1)] = 1.0, 0.0  # the new token
    check_row(model, caches, t, (weight @ values) / weight.sum())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("window,query,key", [(300, 512.0, 32768.0), (300, 2048.0, 41000.0), (1500, 8192.0, 50000.0), (300, 32768.0, 32768.0),
                                              (300, 32768.0, 60000.0)])
def test_large_scores(dtype, window, query, key):
    """Scores up to 2^28, where fp32 has steps of 32: the keys that share the largest one count alike and alone, whichever warp
    has them."""
    model, caches = one_head(dtype, window, query)
    k, v = caches[0].k_ring, caches[0].v_ring
    g = torch.Generator(device=DEV).manual_seed(2)
    first = torch.rand(window + 1, generator=g, device=DEV) < 0.1
    k[0, 0, :, 0] = torch.where(first, key, key / 2)
    v.uniform_(0.25, 1.0, generator=g)
    v[..., 0] = 0.0
    t = 2 * window - 3
    first[t % (window + 1)] = False  # (the new token, whose score is 0)
    check_row(model, caches, t, v[0, 0].double()[first].mean(0))

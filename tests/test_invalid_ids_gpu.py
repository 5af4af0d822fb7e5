"""Token ids, labels and positions outside their tables on the one-call paths: the results say so (NaN), and only those that
depend on them; the status word reports it once."""

import pytest
import torch

from titanmac_b200 import HostPipeline, TitanMAC, TitanMACConfig, _native

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def make(dtype=torch.bfloat16, vocab=128):
    cfg = TitanMACConfig(vocab_size=vocab, d_model=128, n_heads=2, n_layers=2, d_ff=256, max_seq_len=64, window_size=16,
                         n_persistent=3, use_block_sparse=False)
    with torch.device(DEV):
        model = TitanMAC(cfg)
    g = torch.Generator(device=DEV).manual_seed(0)
    return model.to(dtype), torch.randint(0, vocab, (2, 30), generator=g, device=DEV)


def reported():
    with pytest.raises(_native.TmwError, match="outside its table"):
        _native.poll_status(torch.device(DEV))
    _native.poll_status(torch.device(DEV))


@pytest.mark.parametrize("bad", [128, -1, 1 << 40, -(1 << 40)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_ids(bad, dtype):
    model, ids = make(dtype)
    ids[1, 5] = bad
    with torch.no_grad():
        logits = model(ids)["logits"]
        assert torch.isfinite(logits[0]).all() and torch.isnan(logits[1, 5:]).all()
        reported()
        last, caches = model.prefill(ids)
        assert torch.isfinite(last[0]).all() and torch.isnan(last[1]).all()
        reported()
        step = model.decode_step(torch.tensor([3, bad], device=DEV), torch.zeros(2, dtype=torch.int32, device=DEV),
                                 model.new_caches(2, DEV, dtype))
        assert torch.isfinite(step[0]).all() and torch.isnan(step[1]).all()
        reported()
    with torch.enable_grad():
        loss = model(ids, labels=ids.clamp(0, 127))["loss"]
        loss.backward()
    assert torch.isnan(loss) and torch.isnan(model.lm_head.weight.grad).any()
    reported()


@pytest.mark.parametrize("bad", [64, -1])
def test_positions(bad):
    model, _ = make()
    pos = torch.tensor([2, bad], dtype=torch.int32, device=DEV)
    step = model.decode_step(torch.tensor([3, 4], device=DEV), pos, model.new_caches(2, DEV, torch.bfloat16))
    assert torch.isfinite(step[0]).all() and torch.isnan(step[1]).all()
    reported()


@pytest.mark.parametrize("bad", [128, -1, -99, 1 << 40])
def test_labels(bad):
    model, ids = make()
    labels = ids.clone()
    labels[1, 5] = bad
    with torch.enable_grad():
        loss = model(ids, labels=labels)["loss"]
        loss.backward()
    assert torch.isnan(loss) and torch.isnan(model.lm_head.weight.grad).any()
    reported()
    labels[1, 5] = -100  # not counted; nor is the first one, which nothing predicts
    labels[0, 0] = bad
    with torch.no_grad():
        assert torch.isfinite(model(ids, labels=labels)["loss"])
    _native.poll_status(torch.device(DEV))


def test_drain_raises():
    model, ids = make()
    pipe = HostPipeline(lambda t: model(t)["logits"], ids.shape, torch.int64, torch.device(DEV))
    out = torch.empty(2, 30, 128, dtype=torch.bfloat16).pin_memory()
    with torch.no_grad():
        pipe.submit(ids.cpu().pin_memory(), out)
        pipe.drain()
        ids[0, 0] = 128
        pipe.submit(ids.cpu().pin_memory(), out)
        with pytest.raises(_native.TmwError):
            pipe.drain()
    assert torch.isnan(out[0]).all() and torch.isfinite(out[1]).all()

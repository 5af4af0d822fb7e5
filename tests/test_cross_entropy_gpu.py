"""``tmw_cross_entropy`` against PyTorch in fp64 on logits that are not ordinary numbers."""

import pytest
import torch
import torch.nn.functional as F

from titanmac_b200 import _native, _train

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
INF = float("inf")


def special(kind, x, labels, n_p):
    """Changes the row of sequence 1 that predicts labels[1, 3]."""
    row = x[1, n_p + 2]
    y = int(labels[1, 3])
    if kind == "nan":
        row[5] = float("nan")
    elif kind == "inf":
        row[(y + 9) % row.numel()] = INF
    elif kind == "inf_label":
        row[y] = INF
    elif kind == "all_inf":
        row[:] = -INF
    elif kind == "masked":      # whole vectors of eight hidden, the label's left
        row[:] = torch.where(torch.arange(row.numel(), device=row.device) // 8 == y // 8, row, -INF)
    elif kind == "masked_first":  # the first vectors of every thread
        row[: row.numel() // 2] = -INF
        labels[1, 3] = row.numel() - 1
    elif kind == "masked_label":
        row[y] = -INF
    elif kind == "lowest":
        row[: row.numel() // 2] = torch.finfo(row.dtype).min
        labels[1, 3] = row.numel() - 1


@pytest.mark.parametrize("kind", ["plain", "nan", "inf", "inf_label", "all_inf", "masked", "masked_first", "masked_label", "lowest"])
@pytest.mark.parametrize("dtype,V", [(torch.bfloat16, 40), (torch.float16, 5000), (torch.bfloat16, 32000)])
def test_logits_that_are_not_ordinary(kind, dtype, V):
    g = torch.Generator(device=DEV).manual_seed(V)
    n_p, B, T = 3, 2, 6
    x = (torch.randn(B, n_p + T, V, generator=g, device=DEV) * 3).to(dtype)
    labels = torch.randint(0, V, (B, T), generator=g, device=DEV)
    labels[0, 2] = -100
    special(kind, x, labels, n_p)
    with torch.enable_grad():  # (other tests may have turned it off)
        a = x.clone().requires_grad_(True)
        loss = _train.shifted_cross_entropy(a, labels, n_p)[1]
        loss.backward()
        b = x.double().requires_grad_(True)
        want = F.cross_entropy(b[:, n_p:-1].reshape(-1, V), labels[:, 1:].reshape(-1), ignore_index=-100)
        want.backward()
    _native.poll_status(torch.device(DEV))
    eps = torch.finfo(dtype).eps  # one rounding of a result that is an fp32 sum (1e-5) of fp32 exponentials
    assert torch.isnan(loss).item() == torch.isnan(want).item() and torch.isinf(loss).item() == torch.isinf(want).item(), (loss, want)
    if torch.isfinite(want):
        assert abs(loss.item() - want.item()) <= (eps + 1e-5) * abs(want.item())
    # the other rows' gradients are what they were; in the changed row NaN where the reference has it
    got, ref = a.grad.double(), b.grad
    rows = torch.ones(B, n_p + T, dtype=torch.bool, device=DEV)
    rows[1, n_p + 2] = False
    scale = 1.0 / 9  # nine counted rows: an entry is at most that
    assert ((got - ref)[rows].abs() <= eps * ref[rows].abs() + 1e-5 * scale + torch.finfo(dtype).tiny).all()
    assert torch.equal(torch.isnan(got[~rows]).any(), torch.isnan(ref[~rows]).any())
    if not torch.isnan(ref[~rows]).any():
        assert ((got - ref)[~rows].abs() <= eps * ref[~rows].abs() + 1e-5 * scale + torch.finfo(dtype).tiny).all()

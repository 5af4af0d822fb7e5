"""Forward cores at the edges of their tiles: the register-tiled fp32 kernel (32 rows x 64 keys, two groups of threads that
take the key tiles in turn) and the kernel of the block-sparse class's persistent rows (16 rows, keys split over a cluster)."""

import math

import pytest
import torch

from oracle import block_sparse_oracle as bo
from oracle import windowed_oracle as wo
from titanmac_b200 import _native

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dh", [64, 128])
@pytest.mark.parametrize("L,w,n_p", [
    (1, 0, 0), (32, 31, 0), (33, 0, 1),      # one key, one full tile of rows, self-only windows behind a persistent key
    (64, 63, 0), (65, 64, 1), (129, 500, 0), # one and two key tiles exactly, and one key more
    (200, 40, 64), (230, 100, 130),          # rows that see persistent keys only, one tile and more of them
])
def test_fp32_core_at_tile_edges(dh, L, w, n_p):
    q, k, v = wo.qkv_inputs(2, 3, L, dh, seed=dh + L)
    ref = wo.attention_core_dense(q, k, v, w, n_p)
    lse = torch.empty(2, 3, L, device=DEV)
    o = _native.prefill(q.to(DEV), k.to(DEV), v.to(DEV), w, n_p, lse=lse)
    assert (o.cpu() - ref).abs().max().item() <= 1e-5
    s = (q.double() @ k.double().transpose(-1, -2)) / dh ** 0.5
    s = s.masked_fill(~wo.band_mask(L, w, n_p), float("-inf"))
    assert (lse.cpu() - torch.logsumexp(s, -1) / math.log(2.0)).abs().max().item() <= 2e-5


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 2e-2), (torch.float16, 2e-2)])
@pytest.mark.parametrize("dh,L,w,block,n_p", [
    (64, 40, 64, 64, 1), (64, 257, 64, 64, 16), (64, 300, 128, 32, 17),   # 1, 16 and 17 persistent rows
    (128, 500, 96, 32, 33), (128, 129, 64, 64, 128), (128, 1040, 512, 64, 16),
])
def test_block_sparse_core_with_persistent_rows(dtype, tol, dh, L, w, block, n_p):
    q, k, v = (t.to(dtype) for t in wo.qkv_inputs(2, 3, L, dh, seed=dh + L))
    ref = bo.attention_core(q.float(), k.float(), v.float(), w, block, n_p)
    o = _native.prefill(q.to(DEV), k.to(DEV), v.to(DEV), w, n_p, window_block=block)
    _native.poll_status()
    assert (o.float().cpu() - ref).abs().max().item() <= tol


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_persistent_rows_of_many_sequences(dtype):
    """As many sequences as fit the chip three CTAs to an SM (here four to a sequence), and one more: a sequence's rows are the same
    in both launches, bit for bit; one of them against the oracle, tolerance as above."""
    most = 3 * torch.cuda.get_device_properties(0).multi_processor_count // 4
    q, k, v = (t.to(dtype) for t in wo.qkv_inputs(most + 1, 1, 520, 64, seed=3))
    many = _native.prefill(q.to(DEV), k.to(DEV), v.to(DEV), 40, 16, window_block=32)
    few = _native.prefill(q[:most].to(DEV), k[:most].to(DEV), v[:most].to(DEV), 40, 16, window_block=32)
    _native.poll_status()
    assert torch.equal(many[:most], few)
    ref = bo.attention_core(q[-1:].float(), k[-1:].float(), v[-1:].float(), 40, 32, 16)
    assert (many[-1:].float().cpu() - ref).abs().max().item() <= 2e-2


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("L,w,n_p,block", [
    (700, 511, 16, 0), (700, 512, 16, 0),     # either side of the rule: the general body alone, whole tiles on their own
    (641, 512, 0, 0), (1100, 513, 128, 0),    # no persistent keys: the first tile sets the maximum; a ragged left edge
    (1500, 700, 5, 64), (129, 4000, 16, 0),   # block-granular left edge; a window wider than the sequence
])
@pytest.mark.parametrize("spread", [1.0, 8.0])
def test_wide_heads_with_long_windows(dtype, L, w, n_p, block, spread):
    """Whole key tiles without a mask (head_dim 128, windows from 512 on).  ``spread`` 8 makes scores of up to about 100, whose
    running maximum grows by more than 2^8 inside such tiles.  Tolerance: probabilities rounded to bf16 (2^-9) weight values
    of up to 5."""
    q, k, v = (t.to(dtype) for t in wo.qkv_inputs(1, 2, L, 128, seed=L + w))
    q = (q.float() * spread).to(dtype)
    ref = (bo.attention_core(q.float(), k.float(), v.float(), w, block, n_p) if block
           else wo.attention_core_dense(q.float(), k.float(), v.float(), w, n_p))
    o = _native.prefill(q.to(DEV), k.to(DEV), v.to(DEV), w, n_p, window_block=block)
    _native.poll_status()
    assert (o.float().cpu() - ref).abs().max().item() <= 2e-2


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_whole_key_tiles_either_side_of_the_rule(dtype):
    """As many sequences of 6 query tiles and two heads as make four tiles to an SM (whole key tiles on their own), and more (the general
    body): the same sums, so a sequence's rows are the same, bit for bit; one of them against the oracle, tolerance as above."""
    most = 4 * torch.cuda.get_device_properties(0).multi_processor_count // 12
    q, k, v = (t.to(dtype) for t in wo.qkv_inputs(most + 2, 2, 700, 128, seed=5))
    many = _native.prefill(q.to(DEV), k.to(DEV), v.to(DEV), 512, 16)
    few = _native.prefill(q[:most].to(DEV), k[:most].to(DEV), v[:most].to(DEV), 512, 16)
    _native.poll_status()
    assert torch.equal(many[:most], few)
    ref = wo.attention_core_dense(q[-1:].float(), k[-1:].float(), v[-1:].float(), 512, 16)
    assert (many[-1:].float().cpu() - ref).abs().max().item() <= 2e-2

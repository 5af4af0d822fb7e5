"""The library's tensor-core linear layer (tmw_linear, through the C ABI) against PyTorch in fp32 on the same
bf16-rounded operands: the shapes of the module's projections and of the block's MLP at prefill and decode size,
ragged sizes, bias and the exact-GELU epilogue."""

import pytest
import torch

from titanmac_b200 import _native

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def reference(x, w, b, gelu):
    y = torch.nn.functional.linear(x.float(), w.float(), None if b is None else b.float())
    return torch.nn.functional.gelu(y) if gelu else y


def run_case(m, n, k, bias, gelu, dtype=torch.bfloat16, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    x = torch.randn(m, k, generator=g, device=DEV).to(dtype)
    w = (torch.randn(n, k, generator=g, device=DEV) * 0.05).to(dtype)
    b = (torch.randn(n, generator=g, device=DEV) * 0.5).to(dtype) if bias else None
    y = _native.linear(x, w, b, gelu=gelu)
    _native.poll_status(torch.device(DEV))
    ref = reference(x, w, b, gelu)
    # one rounding of the result to 16 bits on top of fp32 accumulation in a different order
    tol = (2 ** -8 if dtype == torch.bfloat16 else 2 ** -10) * max(1.0, ref.abs().max().item()) + 1e-3
    err = (y.float() - ref).abs().max().item()
    assert y.shape == (m, n) and y.dtype == dtype
    assert err <= tol, f"m={m} n={n} k={k} bias={bias} gelu={gelu}: observed max-abs error {err:.3e} > {tol:.3e}"


@pytest.mark.parametrize("m", [256, 32896])
@pytest.mark.parametrize("n,k,bias,gelu", [
    (1920, 640, False, False),   # QKV projection
    (640, 640, False, False),    # output projection
    (2560, 640, True, True),     # MLP fc1 + bias + GELU
    (640, 2560, True, False),    # MLP fc2 + bias
])
def test_layer_shapes(m, n, k, bias, gelu):
    run_case(m, n, k, bias, gelu)


@pytest.mark.parametrize("m,n,k", [(1, 8, 8), (127, 136, 72), (129, 264, 200), (300, 50000, 640), (515, 128, 64),
                                   (700, 40, 64), (1000, 1944, 128), (513, 24, 640)])  # narrow last tiles of the pair kernel
def test_ragged_sizes(m, n, k):
    run_case(m, n, k, True, False, seed=m)
    run_case(m, n, k, False, True, seed=m + 1)


@pytest.mark.parametrize("m,n,k", [(8320, 640, 72), (8321, 616, 128), (6144, 1000, 64), (16416, 328, 72)])
def test_column_tiles_narrower_than_256(m, n, k):
    """Few waves of row bands: the pair kernel cuts N into tiles of 128 to 224 columns."""
    run_case(m, n, k, True, False, seed=m)
    run_case(m, n, k, False, True, dtype=torch.float16, seed=n)


@pytest.mark.parametrize("m,n,k", [(12544, 4096, 64), (12545, 4104, 72), (2300, 4360, 4096), (2048, 4096, 8200)])
def test_wide_outputs_in_groups_of_row_bands(m, n, k):
    """Sixteen column tiles and more: 49 and 50 bands in groups of 48, 9 in one of 16, 8 of the least size."""
    run_case(m, n, k, False, False, seed=m + n)


def test_fp16_and_strided_input():
    run_case(200, 320, 128, True, True, dtype=torch.float16)
    g = torch.Generator(device=DEV).manual_seed(9)
    big = torch.randn(64, 3, 256, generator=g, device=DEV).to(torch.bfloat16)
    x = big[:, 1]  # rows 768 elements apart
    w = (torch.randn(160, 256, generator=g, device=DEV) * 0.05).to(torch.bfloat16)
    y = _native.linear(x, w)
    assert (y.float() - reference(x, w, None, False)).abs().max().item() <= 2e-2


@pytest.mark.parametrize("m,n", [(300, 648), (8320, 664), (97, 40)])
@pytest.mark.parametrize("shift", [0, 8])
def test_output_rows_off_the_32_byte_boundary(m, n, shift):
    """Rows of 16 n + 8 values, or an output 16 bytes into its allocation, go out in halves of sectors; what surrounds them
    stays untouched.  Tolerance: one rounding of values below 8 to bf16, and the order of 128 fp32 sums."""
    g = torch.Generator(device=DEV).manual_seed(m + n)
    x = torch.randn(m, 128, generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn(n, 128, generator=g, device=DEV) * 0.05).to(torch.bfloat16)
    room = torch.full((m * n + 32,), 7.0, device=DEV, dtype=torch.bfloat16)
    out = room[shift:shift + m * n].view(m, n)
    _native.linear(x, w, out=out)
    assert (out.float() - reference(x, w, None, False)).abs().max().item() <= 2 ** -6 + 1e-3
    assert (room[:shift] == 7).all() and (room[shift + m * n:] == 7).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,n", [(33, 8), (97, 40), (300, 648), (257, 1920), (8320, 664), (2060, 2568)])
def test_bias_and_gelu_of_rows_off_the_32_byte_boundary(m, n, dtype):
    """Lanes take their columns eight further on there: the result 16 bytes into its allocation is bit for bit the one at its start,
    and that within one rounding of fp32 (tolerance as in run_case)."""
    g = torch.Generator(device=DEV).manual_seed(m + n)
    x = torch.randn(m, 128, generator=g, device=DEV).to(dtype)
    w = (torch.randn(n, 128, generator=g, device=DEV) * 0.05).to(dtype)
    b = (torch.randn(n, generator=g, device=DEV) * 0.5).to(dtype)
    ref = reference(x, w, b, True)
    tol = (2 ** -8 if dtype == torch.bfloat16 else 2 ** -10) * max(1.0, ref.abs().max().item()) + 1e-3
    outs = []
    for shift in (0, 8):
        room = torch.full((m * n + 32,), 7.0, device=DEV, dtype=dtype)
        out = room[shift:shift + m * n].view(m, n)
        _native.linear(x, w, b, gelu=True, out=out)
        _native.poll_status(torch.device(DEV))
        assert (out.float() - ref).abs().max().item() <= tol
        assert (room[:shift] == 7).all() and (room[shift + m * n:] == 7).all()
        outs.append(out)
    assert torch.equal(*outs)


def test_output_off_the_16_byte_boundary_is_refused():
    x, w = torch.zeros(300, 64, device=DEV, dtype=torch.bfloat16), torch.zeros(64, 64, device=DEV, dtype=torch.bfloat16)
    room = torch.zeros(300 * 64 + 8, device=DEV, dtype=torch.bfloat16)
    with pytest.raises(_native.TmwError):
        _native.linear(x, w, out=room[4:4 + 300 * 64].view(300, 64))


def test_rejects_what_it_cannot_do():
    x = torch.zeros(4, 12, device=DEV, dtype=torch.bfloat16)
    w = torch.zeros(8, 12, device=DEV, dtype=torch.bfloat16)
    with pytest.raises(TypeError):
        _native.linear(x, w)  # k not a multiple of 8
    with pytest.raises(TypeError):
        _native.linear(torch.zeros(4, 16, device=DEV), torch.zeros(8, 16, device=DEV))  # fp32

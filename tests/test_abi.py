"""The C-ABI library loads, exports exactly what include/tmw.h declares, and its host-side
argument checks answer without touching a GPU (no compute call is made here)."""

import ctypes
import os
import re
import subprocess
import tempfile

import pytest

from conftest import ROOT
from titanmac_b200 import _native

HEADER = os.path.join(ROOT, "include", "tmw.h")


def declared_symbols():
    text = open(HEADER).read()
    return sorted(set(re.findall(r"TMW_API[^;()]*?\b(tmw_[a-z_0-9]+)\s*\(", text)))


def test_header_binding_and_exports_agree():
    declared = declared_symbols()
    assert declared, "no TMW_API declarations found"
    assert declared == sorted(_native.SIGNATURES)
    out = subprocess.run(["nm", "-D", "--defined-only", _native.LIB_PATH], capture_output=True, text=True, check=True)
    exported = sorted(line.split()[-1] for line in out.stdout.splitlines() if " T tmw_" in line)
    assert exported == declared
    lib = _native.lib()
    for name in declared:
        assert getattr(lib, name) is not None


def test_struct_layouts_match_the_header():
    src = r"""
    #include <stdio.h>
    #include <stddef.h>
    #include "tmw.h"
    int main(void) {
        printf("%zu %zu %zu %zu %zu\n", sizeof(tmw_prefill_desc), offsetof(tmw_prefill_desc, scale),
               offsetof(tmw_prefill_desc, q_stride), offsetof(tmw_prefill_desc, o_stride),
               offsetof(tmw_prefill_desc, k_pos0));
        printf("%zu %zu %zu %zu\n", sizeof(tmw_cache_desc), offsetof(tmw_cache_desc, k_ring),
               offsetof(tmw_cache_desc, v_pers), offsetof(tmw_cache_desc, scale));
        printf("%zu %zu %zu %zu\n", sizeof(tmw_linear_desc), offsetof(tmw_linear_desc, epilogue),
               offsetof(tmw_linear_desc, lda), offsetof(tmw_linear_desc, ldc));
        return 0;
    }
    """
    with tempfile.TemporaryDirectory() as d:
        c = os.path.join(d, "t.c")
        open(c, "w").write(src)
        exe = os.path.join(d, "t")
        subprocess.run(["gcc", "-I", os.path.join(ROOT, "include"), c, "-o", exe], check=True)
        lines = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split("\n")
    P, C = _native.PrefillDesc, _native.CacheDesc
    assert [int(v) for v in lines[0].split()] == [ctypes.sizeof(P), P.scale.offset, P.q_stride.offset,
                                                  P.o_stride.offset, P.k_pos0.offset]
    assert [int(v) for v in lines[1].split()] == [ctypes.sizeof(C), C.k_ring.offset, C.v_pers.offset, C.scale.offset]
    G = _native.LinearDesc
    assert [int(v) for v in lines[2].split()] == [ctypes.sizeof(G), G.epilogue.offset, G.lda.offset, G.ldc.offset]


def test_version_and_error_text():
    lib = _native.lib()
    assert lib.tmw_version() == 100
    assert lib.tmw_strerror(0) == b"ok"
    for code in range(-8, 0):
        assert lib.tmw_strerror(code) not in (b"ok", b"unknown status")
    assert lib.tmw_strerror(-99) == b"unknown status"


def _desc(**kw):
    d = _native.PrefillDesc()
    d.dtype, d.algo = _native.TMW_BF16, 0
    d.batch, d.heads, d.head_dim = 1, 1, 64
    d.q_rows = d.k_rows = 128
    d.window, d.n_persistent, d.q_pos0, d.k_pos0 = 16, 4, 0, 4
    for i, s in enumerate((0, 64, 64)):
        d.q_stride[i] = d.k_stride[i] = d.v_stride[i] = d.o_stride[i] = s
    for k, v in kw.items():
        setattr(d, k, v)
    return d


@pytest.mark.parametrize("kw,expected", [
    (dict(window=-1), _native.TMW_ERR_NEGATIVE_WINDOW),
    (dict(n_persistent=128, k_pos0=128), _native.TMW_ERR_PERSISTENT_GE_LEN),
    (dict(n_persistent=200, k_pos0=200), _native.TMW_ERR_PERSISTENT_GE_LEN),
    (dict(dtype=7), _native.TMW_ERR_UNSUPPORTED),
    (dict(k_pos0=2), _native.TMW_ERR_INVALID_ARGUMENT),
    (dict(q_rows=-1), _native.TMW_ERR_INVALID_ARGUMENT),
    (dict(algo=9), _native.TMW_ERR_INVALID_ARGUMENT),
    (dict(q_pos0=300), _native.TMW_ERR_KEY_RANGE),          # queries past the last key
    (dict(q_pos0=60, k_pos0=50), _native.TMW_ERR_KEY_RANGE),  # window starts before the first held key
])
def test_prefill_rejects_bad_descriptors_on_the_host(kw, expected):
    d = _desc(**kw)
    fake = ctypes.c_void_p(0x1000)  # never dereferenced: validation fails first
    assert _native.lib().tmw_prefill(ctypes.byref(d), fake, fake, fake, fake, None) == expected


def test_prefill_rejects_null_misaligned_and_odd_strides():
    lib = _native.lib()
    ok = ctypes.c_void_p(0x1000)
    d = _desc()
    assert lib.tmw_prefill(None, ok, ok, ok, ok, None) == _native.TMW_ERR_INVALID_ARGUMENT
    assert lib.tmw_prefill(ctypes.byref(d), None, ok, ok, ok, None) == _native.TMW_ERR_INVALID_ARGUMENT
    assert lib.tmw_prefill(ctypes.byref(d), ctypes.c_void_p(0x1004), ok, ok, ok, None) == _native.TMW_ERR_INVALID_ARGUMENT
    d = _desc()
    d.k_stride[2] = 63
    assert lib.tmw_prefill(ctypes.byref(d), ok, ok, ok, ok, None) == _native.TMW_ERR_INVALID_ARGUMENT
    # an empty problem is fine and launches nothing
    assert lib.tmw_prefill(ctypes.byref(_desc(batch=0)), None, None, None, None, None) == _native.TMW_OK


def test_cache_entry_points_reject_bad_arguments_on_the_host():
    lib = _native.lib()
    assert lib.tmw_cache_ring_bytes(_native.TMW_BF16, 256, 10, 64, 512) == 256 * 10 * 513 * 64 * 2
    assert lib.tmw_cache_ring_bytes(_native.TMW_F32, 2, 3, 16, 0) == 2 * 3 * 1 * 16 * 4
    assert lib.tmw_cache_ring_bytes(9, 1, 1, 64, 4) == 0
    c = _native.CacheDesc()
    c.dtype, c.batch, c.heads, c.head_dim, c.window, c.n_persistent = _native.TMW_BF16, 1, 1, 64, -2, 0
    s3 = (ctypes.c_int64 * 3)(0, 64, 64)
    s2 = (ctypes.c_int64 * 2)(64, 64)
    ok = ctypes.c_void_p(0x1000)
    assert lib.tmw_cache_fill(ctypes.byref(c), ok, ok, s3, s3, 4, 0, None) == _native.TMW_ERR_NEGATIVE_WINDOW
    c.window, c.head_dim = 4, 48
    assert lib.tmw_decode(ctypes.byref(c), ok, ok, ok, ok, s2, s2, s2, ok, None) == _native.TMW_ERR_UNSUPPORTED
    c.head_dim = 64  # rings are NULL
    assert lib.tmw_decode(ctypes.byref(c), ok, ok, ok, ok, s2, s2, s2, ok, None) == _native.TMW_ERR_INVALID_ARGUMENT


def test_split_decode_scratch_size_and_argument_checks():
    lib = _native.lib()
    c = _native.CacheDesc()
    c.dtype, c.batch, c.heads, c.head_dim, c.window, c.n_persistent = _native.TMW_BF16, 32, 10, 64, 512, 0
    c.k_ring = c.v_ring = 0x1000
    assert lib.tmw_decode_split_scratch_bytes(ctypes.byref(c), 4) == 32 * 10 * 4 * (64 + 2) * 4 + 32 * 10 * 4
    assert lib.tmw_decode_split_scratch_bytes(ctypes.byref(c), 0) == 0
    assert lib.tmw_decode_split_scratch_bytes(ctypes.byref(c), _native.MAX_DECODE_SPLITS + 1) == 0
    s2 = (ctypes.c_int64 * 2)(640, 64)
    ok = ctypes.c_void_p(0x1000)
    args = (ctypes.byref(c), ok, ok, ok, ok, s2, s2, s2, ok)
    assert lib.tmw_decode_split(*args, 0, ok, 1 << 30, None) == _native.TMW_ERR_INVALID_ARGUMENT   # splits
    assert lib.tmw_decode_split(*args, 4, None, 1 << 30, None) == _native.TMW_ERR_INVALID_ARGUMENT  # no scratch
    assert lib.tmw_decode_split(*args, 4, ok, 1024, None) == _native.TMW_ERR_TOO_LARGE            # scratch too small


def test_decode_step_sizes_the_library_refuses():
    """No workspace, and so no call, beyond what every kernel of the step takes (the check is the same in both)."""
    def workspace(**more):
        sizes = dict(dtype=_native.TMW_BF16, batch=3, layers=1, d_model=4096, heads=32, head_dim=128, d_ff=64, window=8,
                     vocab=16, max_positions=4, eps=1e-5)
        return _native.lib().tmw_decode_step_workspace(ctypes.byref(_native.StackDesc(**dict(sizes, **more))))

    assert workspace() > 0 and workspace(batch=65535) > 0
    assert workspace(d_model=5120, heads=40) == 0 and workspace(batch=65536) == 0
    assert workspace(head_dim=32, heads=128) == 0 and workspace(d_ff=48) == 0
    # a long window over few (sequence, head) pairs is split over more CTAs than a cluster holds, through the workspace
    few = dict(batch=1, d_model=640, heads=10, head_dim=64)
    assert workspace(**few, window=4095) > workspace(**few, window=4094) == workspace(**few)
    assert workspace(**dict(few, batch=64), window=4095) == workspace(**dict(few, batch=64))


def test_scratch_of_a_training_step_follows_its_size():
    """No room for split products where the rows are too few to be cut; never more than 24 MiB a product."""
    lib = _native.lib()

    def module(rows, dim=128):
        d = _native.AttentionDesc(_native.TMW_BF16, 1, rows, dim // 64, 64, 16, 3, 0, 0, 0.0)
        return lib.tmw_attention_train_scratch(ctypes.byref(d)), 4 * rows * dim * 2

    def stack(tokens, dim=128):
        d = _native.StackDesc(dtype=_native.TMW_BF16, batch=1, layers=2, d_model=dim, heads=dim // 64, head_dim=64, d_ff=2 * dim,
                              window=16, n_persistent=0, vocab=512, max_positions=tokens, eps=1e-5)
        return lib.tmw_stack_train_scratch(ctypes.byref(d), tokens), tokens * dim * 2 * (3 + 2 + 3)

    for size in (module, stack):
        nbytes, activations = size(128)
        assert activations <= nbytes <= 4 * activations + (1 << 20)
        nbytes, activations = size(100000, 1024)
        assert activations + (8 << 20) <= nbytes <= 4 * activations + (200 << 20)


def test_training_backward_checks_where_gradients_go_on_the_host():
    """A missing or misaligned gradient is refused before anything is launched: products write 16 bytes at a time, sums of partial
    results 8.  Optional entries (biases, filters) may be NULL."""
    lib, tokens = _native.lib(), 64
    ok = 0x1000  # never dereferenced: validation fails first
    d = _native.StackDesc(dtype=_native.TMW_BF16, batch=1, layers=2, d_model=128, heads=2, head_dim=64, d_ff=256, window=16,
                          n_persistent=4, vocab=512, max_positions=tokens, block_size=16, conv_taps=4, eps=1e-5,
                          embed_tokens=ok, embed_positions=ok, persistent=ok, norm=ok, head=ok)
    nbytes = lib.tmw_stack_train_scratch(ctypes.byref(d), tokens)
    blocks = (_native.Block * 2)()
    for b in blocks:
        b.norm_attn = b.w_qkv = b.w_out = b.norm_mlp = b.w_fc1 = b.w_fc2 = b.conv_q = b.conv_k = b.conv_v = ok

    def refused(layer=None, name=None, at=None, saved=ok):
        grads, block_grads = _native.StackGrads(*[ok] * 5), (_native.BlockGrads * 2)()
        for g in block_grads:
            g.norm_attn = g.w_qkv = g.w_out = g.norm_mlp = g.w_fc1 = g.w_fc2 = ok
        if name is not None:
            setattr(grads if layer is None else block_grads[layer], name, at)
        return lib.tmw_stack_train_backward(ctypes.byref(d), blocks, ctypes.byref(grads), block_grads, ok, tokens, ok, saved, ok, nbytes,
                                            None) == _native.TMW_ERR_INVALID_ARGUMENT

    for name in ("embed_tokens", "head", "embed_positions", "persistent"):
        assert refused(None, name, None) and refused(None, name, ok + 8), name
    assert refused(None, "norm", None) and refused(None, "norm", ok + 4)
    for layer in range(2):
        for name in ("w_qkv", "w_out", "w_fc1", "w_fc2"):
            assert refused(layer, name, None) and refused(layer, name, ok + 8), name
        for name in ("norm_attn", "norm_mlp"):
            assert refused(layer, name, None) and refused(layer, name, ok + 4), name
        for name in ("b_fc1", "b_fc2", "conv_q", "conv_k", "conv_v"):
            assert refused(layer, name, ok + 4), name
    assert refused(saved=ok + 8)

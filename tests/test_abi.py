"""The shared library loads on a CPU-only box and exports every symbol include/et_b200.h
declares; host-side validators and argument checks work without a GPU."""
import ctypes
import os
import re

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared():
    src = open(os.path.join(ROOT, "include", "et_b200.h")).read()
    src = re.sub(r"/\*.*?\*/", "", src, flags=re.S)
    return sorted(set(re.findall(r"\b(et_[a-z0-9_]+)\s*\(", src)))


def test_header_symbols_are_exported(et):
    lib = et.lib()
    declared = _declared()
    assert len(declared) >= 25
    for name in declared:
        assert hasattr(lib, name), f"{name} is declared in et_b200.h but not exported"
    assert sorted(et.ABI_SYMBOLS) == declared


def test_status_strings(et):
    lib = et.lib()
    assert lib.et_status_string(0) == b"ok"
    for code in range(-8, 0):
        assert lib.et_status_string(code) not in (b"ok", b"unknown status")
    assert lib.et_built_for_sm() == 100


def test_missing_library_fails_loudly(et, monkeypatch):
    monkeypatch.setattr(et, "_lib", None)
    monkeypatch.setattr(et, "LIB_PATH", "/nonexistent/libet_b200.so")
    with pytest.raises(et.EtError):
        et.lib()


def _p(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def test_validate_tile_mat(et):
    lib = et.lib()
    w = et.synth.prune_tiles(et.synth.normal(1, 1, (64, 96), 1.0), 1, 2, 0.5)
    rp, ro, tiles = et.synth.dense_to_tile(w)
    assert lib.et_validate_tile_mat(_p(rp), _p(ro), len(ro), 96, 64) == 0
    bad = ro.copy()
    bad[0] = 6  # column block out of range (96 / 16 = 6 blocks)
    assert lib.et_validate_tile_mat(_p(rp), _p(bad), len(ro), 96, 64) == -4
    bad = rp.copy()
    bad[1], bad[2] = bad[2], bad[1] if rp[1] != rp[2] else bad[1] + 1
    assert lib.et_validate_tile_mat(_p(bad), _p(ro), len(ro), 96, 64) == -4
    assert lib.et_validate_tile_mat(_p(rp), _p(ro), len(ro) - 1, 96, 64) == -4
    assert lib.et_validate_tile_mat(_p(rp), _p(ro), len(ro), 100, 64) == -3
    assert lib.et_validate_tile_mat(None, _p(ro), len(ro), 96, 64) == -1


def test_validate_lists_1x16_csr(et):
    lib = et.lib()
    ids = np.array([0, 3, 9], np.int32)
    assert lib.et_validate_id_list(_p(ids), 3, 10, 1) == 0
    assert lib.et_validate_id_list(_p(ids), 3, 9, 1) == -4
    assert lib.et_validate_id_list(_p(ids[::-1].copy()), 3, 10, 1) == -4
    assert lib.et_validate_id_list(_p(ids[::-1].copy()), 3, 10, 0) == 0
    w = et.synth.prune_1x16(et.synth.normal(2, 1, (32, 64), 1.0), 2, 2, 0.7)
    ti, ri, data = et.synth.dense_to_1x16(w)
    assert lib.et_validate_1x16(_p(ti), _p(ri), len(ri), 64, 32) == 0
    bad = ri.copy()
    bad[0] += 16
    assert lib.et_validate_1x16(_p(ti), _p(bad), len(ri), 64, 32) == -4
    ip, ix, dv = et.synth.dense_to_csr(w)
    assert lib.et_validate_csr(_p(ip), _p(ix), len(ix), 64, 32) == 0
    bad = ix.copy()
    bad[-1] = 64
    assert lib.et_validate_csr(_p(ip), _p(bad), len(ix), 64, 32) == -4


def test_argument_checks_need_no_gpu(et):
    """Null pointers and bad sizes are refused before any CUDA call."""
    lib = et.lib()
    assert lib.et_linear_dense_fwd(None, None, None, None, 4, 16, 16, 0, None) == -1
    assert lib.et_linear_dense_fwd(None, None, None, None, 4, 20, 16, 0, None) == -3
    assert lib.et_skip_layernorm_fwd(None, None, None, None, None, 1, 8, None) == -1
    assert lib.et_encoder_layer_workspace_bytes(None, 1, 1) == 0


def test_peer_exchange_argument_checks(et):
    """The head-parallel exchange entry points reject bad arguments before touching a device."""
    lib = et.lib()
    lib.et_peer_buffer_bytes.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_int,
                                         ctypes.POINTER(ctypes.c_size_t)]
    n = ctypes.c_size_t(0)
    assert lib.et_peer_buffer_bytes(8, 4096, 768, ctypes.byref(n)) == 0
    # partial + y + two output buffers of T x hidden fp16, plus the flag words
    assert n.value >= 4 * 4096 * 768 * 2 and n.value < 4 * 4096 * 768 * 2 + 4096
    assert lib.et_peer_buffer_bytes(17, 4096, 768, ctypes.byref(n)) == -1
    assert lib.et_peer_buffer_bytes(8, 0, 768, ctypes.byref(n)) == -1
    bufs = (ctypes.c_void_p * 2)(0x1000, 0x2000)
    # world out of range, rank out of range, a null buffer, an odd hidden size, misalignment
    assert lib.et_hp_signal_partial_fwd(bufs, 0, 17, 128, 768, 1, None) == -1
    assert lib.et_hp_signal_partial_fwd(bufs, 2, 2, 128, 768, 1, None) == -1
    assert lib.et_hp_signal_partial_fwd((ctypes.c_void_p * 2)(0x1000, None), 0, 2, 128, 768, 1, None) == -1
    assert lib.et_hp_signal_partial_fwd(bufs, 0, 2, 128, 772, 1, None) == -3
    assert lib.et_hp_signal_partial_fwd((ctypes.c_void_p * 2)(0x1000, 0x2010), 0, 2, 128, 768, 1, None) == -2
    assert lib.et_hp_allgather_rows_fwd(bufs, 0, 2, 128, 768, 1, 2, None) == -1
    assert lib.et_peer_buffer_open(None, None) == -1


def test_attention_fuse_o_single_launch_argument_checks(et):
    """The one-kernel attention + output projection rejects bad arguments before touching a
    device (error codes of include/et_b200.h: -1 invalid argument, -2 alignment, -3 shape)."""
    lib = et.lib()
    fn = lib.et_attention_fuse_o_single_launch_fwd
    P = ctypes.c_void_p
    fn.argtypes = [P, P, P, P, P, P, P, P, ctypes.c_int, P, P] + [ctypes.c_int] * 10 + [P, ctypes.c_float, P]
    ok = dict(Q=0x1000, K=0x2000, V=0x3000, mask=None, Z=0x4000, rp=0x5000, ro=0x6000, tiles=0x7000,
              nnz=10, bias=None, out=0x8000, batch=1, seq=128, nhead=12, dh_qk=64, dh_v=64, ldq=768,
              ldk=768, ldv=768, emdim=768, mask_kind=0, vl=None, scale=0.125, stream=None)

    def call(**kw):
        a = dict(ok, **kw)
        return fn(*[a[k] for k in ok])

    assert call(Z=None) == -1 and call(out=None) == -1
    assert call(Q=None) == -1 and call(ro=None) == -1
    assert call(mask_kind=7) == -1
    assert call(mask_kind=2) == -1          # padding mask without lengths
    assert call(scale=0.0) == -1
    assert call(dh_qk=40) == -3             # head width not a multiple of 16
    assert call(ldq=760) == -3              # row pitch narrower than the heads
    assert call(emdim=770) == -3
    assert call(Q=0x1008) == -2



def _layer_desc(et, **pointers):
    """A dense 768-wide layer whose pointers are made up: for calls that must be refused on the host."""
    d = et.EncoderLayerDesc()
    for i, (lin, inn, out) in enumerate(((d.qkv, 768, 2304), (d.o, 768, 768), (d.ffn1, 768, 3072),
                                         (d.ffn2, 3072, 768))):
        lin.in_, lin.out, lin.weight, lin.bias = inn, out, 0x100000 * (i + 1), 0x1000 * (i + 1)
    for i, name in enumerate(("ln1_gamma", "ln1_beta", "ln2_gamma", "ln2_beta")):
        setattr(d, name, 0x10000 * (i + 1))
    d.hidden, d.nhead, d.kdim, d.vdim, d.ff, d.act = 768, 12, 768, 768, 3072, 2
    for k, v in pointers.items():
        setattr(d, k, v)
    return d


def test_misaligned_layer_tensors_are_refused_before_a_launch(et):
    """The layer's kernels move x, its output and the all-reduced sum in 16-byte pieces: each is checked on
    the host at the entry, before the first kernel."""
    lib = et.lib()
    d = _layer_desc(et)
    P, Z = ctypes.c_void_p, ctypes.c_size_t
    ref, ws, big = ctypes.byref(d), P(0x40000000), Z(1 << 40)
    before = lib.et_launch_count()
    for x, out in ((0x2000008, 0x3000000), (0x2000000, 0x3000008), (0x2000000, 0x3000002)):
        assert lib.et_encoder_layer_fwd(ref, P(x), P(out), 1, 128, 0, None, None, ws, big, None) == -2
        assert lib.et_encoder_ffn_fwd(ref, P(x), P(out), 1, 128, ws, big, None) == -2
        for f32 in (0, 1):
            assert lib.et_encoder_after_attention_fwd(ref, P(0x5000000), f32, P(x), P(out), 1, 128, ws, big,
                                                      None) == -2
    for f32 in (0, 1):
        assert lib.et_encoder_after_attention_fwd(ref, P(0x5000008), f32, P(0x2000000), P(0x3000000), 1, 128,
                                                  ws, big, None) == -2
    assert lib.et_launch_count() == before


def test_partial_sum_layernorm_refuses_misaligned_vectors(et):
    """bias, gamma and beta of a LayerNorm that adds up fp32 sums are read 16 bytes at a time."""
    lib = et.lib()
    P, Z = ctypes.c_void_p, ctypes.c_size_t
    for name in ("ln1_gamma", "ln1_beta"):
        d = _layer_desc(et, **{name: 0x10002})
        assert lib.et_encoder_after_attention_fwd(ctypes.byref(d), P(0x5000000), 1, P(0x2000000), P(0x3000000), 1,
                                                  128, P(0x40000000), Z(1 << 40), None) == -2
    d = _layer_desc(et)
    d.o.bias = 0x1004
    assert lib.et_encoder_after_attention_fwd(ctypes.byref(d), P(0x5000000), 1, P(0x2000000), P(0x3000000), 1, 128,
                                              P(0x40000000), Z(1 << 40), None) == -2


def test_1x16_refuses_more_than_65535_token_blocks(et):
    lib = et.lib()
    P = ctypes.c_void_p
    lib.et_linear_1x16_fwd.argtypes = [P, P, P, ctypes.c_int, P, P, P] + [ctypes.c_int] * 4 + [P]
    args = lambda T: (P(0x1000), P(0x2000), P(0x3000), 4, None, P(0x4000), P(0x5000), T, 64, 64, 0, None)
    assert lib.et_linear_1x16_fwd(*args(65535 * 128 + 1)) == -3


def test_csr_plan_follows_the_stored_values(et):
    """Almost empty weights take the kernel whose work follows what is stored (it was 2 to 5 times as fast there),
    others the expanded tensor-core product, and nothing in between switches back."""
    pays = et.lib().et_debug_csr_rows_pay
    for T, inn, out in ((8192, 1024, 3072), (2048, 3072, 768), (128, 3072, 768), (8192, 4096, 1024), (8192, 768, 768)):
        total = inn * out
        chosen = [pays(T, inn, out, int(total * f)) for f in (0.0, 0.001, 0.01, 0.03, 0.1, 0.5)]
        assert chosen[0] == chosen[1] == 1 and chosen[3:] == [0, 0, 0], (T, inn, out, chosen)
        assert chosen == sorted(chosen, reverse=True)


def test_almost_empty_packed_tiles_stay_on_the_kernel_that_follows_them(et):
    """The expanding kernel takes long K with few output tiles, but not where hardly a tile is stored: its time
    does not fall with them."""
    expands = et.lib().et_debug_tile_packed_expands
    for T, inn, out in ((1, 3072, 768), (1000, 3072, 768), (1000, 4096, 1024), (128, 2048, 512)):
        total = (inn // 16) * (out // 16)
        assert [expands(T, inn, out, int(total * f)) for f in (0.2, 0.1, 0.05, 0.01, 0.001)] == [1, 1, 1, 0, 0]
    assert expands(8192, 3072, 768, 4608) == 0 and expands(128, 768, 3072, 4608) == 0


def test_narrow_gemm_tiles_with_few_tokens(et):
    """Tiles of the GEMM for few output tiles: with up to 64 tokens all CTAs read the same lines of X, so wide
    outputs must not be cut into a hundred of them (1024 -> 4096 took 9.9 us for 6.0 at one token)."""
    width = et.lib().et_debug_gemm_narrow_width
    assert [width(1, n) for n in (512, 768, 1024, 2048, 2304, 3072, 4096)] == [32, 32, 32, 64, 64, 0, 0]
    assert [width(31, n) for n in (1024, 2304, 3072)] == [32, 64, 0]
    assert [width(32, n) for n in (1024, 2304, 3072, 4096)] == [32, 64, 64, 64]
    assert [width(64, n) for n in (768, 2304, 3072)] == [32, 32, 64]
    assert [width(33, n) for n in (2304, 2320)] == [32, 64]
    assert [width(65, n) for n in (768, 3072, 4096)] == [32, 32, 32]
    assert width(385, 768) == 32 and width(128 * 12, 768) == 64 and width(128 * 13, 768) == 0


def test_depth_of_the_fused_projection_ring(et):
    """Five stages where every CTA has an SM to itself, but not beside an additive mask that they would push out
    of the L1 cache (1 x 128 tokens, 12 heads, had gone from 18.4 to 22.2 us)."""
    deep = et.lib().et_debug_qkv_deep
    assert [deep(128, 12, b, 0) for b in (1, 12, 13)] == [1, 1, 0]
    assert [deep(s, 12, 1, 3) for s in (1, 100, 106, 107, 127, 128)] == [1, 1, 1, 0, 0, 0]
    assert [deep(128, 12, b, 3) for b in (2, 3, 12, 13)] == [0, 1, 1, 0]

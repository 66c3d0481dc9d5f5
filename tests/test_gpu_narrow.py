"""The kernels for few row blocks: 128 x 32 / 128 x 64 GEMM tiles, fp32 K slices of tiles up to 128 wide
added up by the LayerNorm, and the deep-ring form of the fused projection + attention; at ragged
sizes and at the edges of the rules that choose them.

The narrow GEMM accumulates K in the order of the wider tiles, so its results are theirs bit for bit;
the encoder layer is compared with the fp32 oracle at the suite's fp16 tolerance."""
import ctypes

import numpy as np
import pytest

from conftest import assert_close

pytestmark = pytest.mark.gpu


def _dev(a, cuda):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).to(cuda)


@pytest.mark.parametrize("T,inn,out,act", [(1, 16, 16, 0), (128, 768, 768, 0), (129, 80, 144, 2),
                                           (300, 1040, 1008, 1), (385, 3072, 80, 2), (64, 64, 3072, 2),
                                           (31, 256, 3072, 0), (33, 1024, 2320, 2)])
def test_narrow_tiles_match_wide_ones(et, cuda, T, inn, out, act):
    import torch
    x = _dev(et.synth.normal_fast(81, 1, (T, inn), 1.0), cuda)
    w = _dev(et.synth.normal_fast(81, 2, (out, inn), 0.05), cuda)
    b = _dev(et.synth.normal_fast(81, 3, (out,), 0.1), cuda)
    L = et.lib()
    ys = []
    try:
        for bn in (0, 32, 64):
            L.et_debug_force_gemm_narrow(ctypes.c_int(bn))
            ys.append(et.linear_dense(x, w, b, act))
            assert et.device_error() == 0
    finally:
        L.et_debug_force_gemm_narrow(ctypes.c_int(-1))
    assert torch.equal(ys[0], ys[1]) and torch.equal(ys[0], ys[2])


@pytest.mark.parametrize("batch,seq,hidden,nhead,ff", [
    (1, 1, 256, 4, 512),       # one token
    (1, 128, 768, 12, 3072),   # one row block: 32-wide tiles, four slices
    (5, 77, 768, 12, 3072),    # ragged row blocks: 64-wide tiles, three slices
    (7, 128, 768, 12, 1536),   # 128-wide tiles
    (12, 128, 1024, 16, 1024),  # the last grid with an SM for every projection CTA is 9 x 16
    (3, 130, 512, 8, 2048),    # sequences longer than a row block
    (2, 50, 1040, 13, 1104),   # nothing a multiple of a tile
])
def test_layer_with_few_row_blocks(et, orc, cuda, batch, seq, hidden, nhead, ff):
    import torch
    w = et.synth.encoder_layer_weights(82, 0, hidden, ff, bias_std=0.02, ln_noise=0.05, fast=True)
    x = et.synth.normal_fast(82, 9, (batch * seq, hidden), 1.0)
    vl = np.array([max(1, seq - 5 * i) for i in range(batch)], dtype=np.int32)
    stack = et.EncoderStack([et.EncoderLayer(w, nhead, et.ACT_GELU, device=cuda)], batch, seq, device=cuda)
    y = stack.forward(_dev(x, cuda), et.MASK_PADDING, None, _dev(vl, cuda)).clone()
    assert et.device_error() == 0
    ref = orc.encoder_layer(x.astype(np.float32), w, batch, seq, nhead, 2, 2, None, vl)
    assert_close(y.float().cpu().numpy(), ref, f"layer {batch}x{seq}x{hidden}")
    assert torch.equal(y, stack.forward(_dev(x, cuda), et.MASK_PADDING, None, _dev(vl, cuda)))
    # and with the fused or the plain Linear + LayerNorm in place of the K slices: the plain one rounds the product
    # to fp16 before the LayerNorm
    et.lib().et_debug_set_narrow_ln(ctypes.c_int(0))
    try:
        other = stack.forward(_dev(x, cuda), et.MASK_PADDING, None, _dev(vl, cuda))
    finally:
        et.lib().et_debug_set_narrow_ln(ctypes.c_int(-1))
    assert et.device_error() == 0
    assert_close(y.float().cpu().numpy(), other.float().cpu().numpy(), f"forms of {batch}x{seq}x{hidden}",
                 rel_tol=1.5e-3)


@pytest.mark.parametrize("batch,seq", [(1, 128), (5, 77)])
def test_layer_with_vectors_off_16_byte_boundaries(et, orc, cuda, batch, seq):
    """bias, gamma and beta of the O projection and FFN2 may lie anywhere: the fused kernel reads them one
    element at a time, and a layer with few row blocks must not lose that to the narrow tiles."""
    import torch
    hidden, nhead, ff = 768, 12, 3072
    w = et.synth.encoder_layer_weights(83, 0, hidden, ff, bias_std=0.02, ln_noise=0.05, fast=True)
    x = et.synth.normal_fast(83, 9, (batch * seq, hidden), 1.0)
    layer = et.EncoderLayer(w, nhead, et.ACT_GELU, device=cuda)
    keep = []

    def shifted(a, by):
        t = torch.zeros(a.size + 8, dtype=torch.float16, device=cuda)
        t[by:by + a.size] = torch.from_numpy(np.ascontiguousarray(a, np.float16)).to(cuda)
        keep.append(t)
        return t.data_ptr() + 2 * by

    for i, n in enumerate(("ln1_gamma", "ln1_beta", "ln2_gamma", "ln2_beta")):
        setattr(layer.desc, n, shifted(w[n.replace("amma", "").replace("eta", "")], i + 1))
    layer.desc.o.bias = shifted(w["bo"], 5)
    layer.desc.ffn2.bias = shifted(w["b2"], 6)
    stack = et.EncoderStack([layer], batch, seq, device=cuda)
    y = stack.forward(_dev(x, cuda)).clone()
    assert et.device_error() == 0
    ref = orc.encoder_layer(x.astype(np.float32), w, batch, seq, nhead, 2, 0, None, None)
    assert_close(y.float().cpu().numpy(), ref, f"shifted vectors {batch}x{seq}")
    # an output off a boundary is refused, and nothing is launched
    before = et.lib().et_launch_count()
    out = torch.zeros(batch * seq * hidden + 8, dtype=torch.float16, device=cuda)[4:4 + batch * seq * hidden]
    ws = torch.empty(et.lib().et_encoder_layer_workspace_bytes(ctypes.byref(layer.desc), batch, seq),
                     dtype=torch.uint8, device=cuda)
    with pytest.raises(et.EtError, match="-2"):
        layer.forward(_dev(x, cuda), out, batch, seq, ws)
    assert et.lib().et_launch_count() == before and et.device_error() == 0

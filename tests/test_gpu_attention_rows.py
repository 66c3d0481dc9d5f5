"""The one-row-per-thread attention kernel (heads of up to 64 features) at its edges: block and
sequence remainders, head widths below a 64-feature atom, every mask kind, rising maxima (rescaled
accumulators), against the oracle and against the kernel that splits a row over two threads."""
import ctypes

import numpy as np
import pytest

from conftest import assert_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,seq,nhead,dh_qk,dh_v", [
    (1, 1, 1, 16, 16), (2, 127, 2, 48, 64), (2, 129, 3, 64, 48), (1, 257, 2, 64, 64),
    (1, 385, 2, 32, 32), (3, 640, 1, 64, 64),
])
@pytest.mark.parametrize("mask_kind", [0, 1, 2, 3])
@pytest.mark.parametrize("std", [1.0, 4.0])
def test_attention_rows(et, orc, cuda, batch, seq, nhead, dh_qk, dh_v, mask_kind, std):
    import torch
    T = batch * seq
    q = et.synth.normal(700 + seq, 1, (T, nhead * dh_qk), std)
    k = et.synth.normal(700 + seq, 2, (T, nhead * dh_qk), std)
    # later keys score higher: the running maximum rises from block to block
    k = (k.astype(np.float32) * (1.0 + np.arange(T) % seq / seq)[:, None]).astype(np.float16)
    v = et.synth.normal(700 + seq, 3, (T, nhead * dh_v), 1.0)
    vl = np.array([(seq * (i + 1)) // 2 + i for i in range(batch)], dtype=np.int32).clip(0, seq)
    vl[0] = 0 if batch > 1 else seq  # a sequence without keys gives zeros
    mask = None
    if mask_kind == 3:
        mask = np.where(et.synth.normal(700, 7, (seq, seq), 1.0).astype(np.float32) > 0.8,
                        -np.inf, 0.0).astype(np.float16)
        mask[0, :] = -np.inf  # a row without keys
    d = lambda a: None if a is None else torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    args = (d(q), d(k), d(v), batch, seq, nhead, dh_qk, dh_v, mask_kind, d(mask),
            d(vl) if mask_kind == 2 else None)
    z = et.attention(*args)
    assert et.device_error() == 0
    L = et.lib()
    L.et_debug_set_attention_rows(ctypes.c_int(0))
    try:
        split = et.attention(*args)
    finally:
        L.et_debug_set_attention_rows(ctypes.c_int(1))
    assert et.device_error() == 0
    # the two differ in the order of the row sums only: one fp16 rounding of values below max |V|
    diff = (z.float() - split.float()).abs().max().item()
    assert diff <= np.abs(v.astype(np.float32)).max() * 2.0 ** -10, diff
    ref = orc.attention(q, k, v, batch, seq, nhead, dh_qk, dh_v, mask_kind, mask,
                        vl if mask_kind == 2 else None)
    assert_close(z.float().cpu().numpy(), ref, f"rows s{seq} m{mask_kind} std{std}")

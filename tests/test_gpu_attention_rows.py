"""The one-row-per-thread attention kernel (heads of up to 64 features) at its edges: block and
sequence remainders, head widths below a 64-feature atom, every mask kind, rising maxima (rescaled
accumulators), against the oracle and against the kernel that splits a row over two threads."""
import ctypes

import numpy as np
import pytest

from conftest import assert_close

pytestmark = pytest.mark.gpu


def _split_rows(et, args):
    """The same call on the kernel that splits a row over two threads."""
    et.lib().et_debug_set_attention_rows(ctypes.c_int(0))
    try:
        z = et.attention(*args)
    finally:
        et.lib().et_debug_set_attention_rows(ctypes.c_int(1))
    assert et.device_error() == 0
    return z


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
    if mask_kind != 3:  # an additive mask takes the split-row kernel either way
        split = _split_rows(et, args)
        # the two differ in the order of the row sums and in how a quarter of the exponentials is computed, both
        # in fp32: one fp16 rounding of values below max |V|
        diff = (z.float() - split.float()).abs().max().item()
        assert diff <= np.abs(v.astype(np.float32)).max() * 2.0 ** -10, diff
    ref = orc.attention(q, k, v, batch, seq, nhead, dh_qk, dh_v, mask_kind, mask,
                        vl if mask_kind == 2 else None)
    assert_close(z.float().cpu().numpy(), ref, f"rows s{seq} m{mask_kind} std{std}")


@pytest.mark.parametrize("batch,seq,nhead,dh_v", [
    (20, 257, 12, 64),  # 720 items, two to three a CTA; outputs through the staging tile
    (20, 257, 12, 48),  # outputs stored directly
    (40, 257, 12, 64),  # 1440 items: more than eight per SM, where causal items are dealt in another order
    (5, 1025, 16, 64),  # items of one to nine blocks of keys
])
@pytest.mark.parametrize("mask_kind", [0, 1, 2])
def test_attention_rows_several_items_a_cta(et, orc, cuda, batch, seq, nhead, dh_v, mask_kind):
    """What a persistent CTA carries from item to item: barrier phases, the rings, Q, S, P and O; and sequences
    without keys between others, which only the softmax warps visit."""
    import torch
    T, dh_qk = batch * seq, 64
    g = torch.Generator(device=cuda)
    g.manual_seed(batch + seq + dh_v)
    rand = lambda n: torch.randn((T, n), generator=g, device=cuda).half()
    q, k, v = rand(nhead * dh_qk), rand(nhead * dh_qk), rand(nhead * dh_v)
    vl = torch.randint(1, seq + 1, (batch,), generator=g, device=cuda, dtype=torch.int32)
    vl[1::3] = 0
    vl[2::4] = seq
    args = (q, k, v, batch, seq, nhead, dh_qk, dh_v, mask_kind, None, vl if mask_kind == 2 else None)
    z = et.attention(*args)
    assert et.device_error() == 0
    assert torch.equal(z, et.attention(*args))
    diff = (z.float() - _split_rows(et, args).float()).abs().max().item()
    assert diff <= v.float().abs().max().item() * 2.0 ** -10, diff
    for b in (0, batch // 2, batch - 1):
        s = slice(b * seq, (b + 1) * seq)
        ref = orc.attention(q[s].cpu().numpy(), k[s].cpu().numpy(), v[s].cpu().numpy(), 1, seq, nhead, dh_qk, dh_v,
                            mask_kind, None, vl[b:b + 1].cpu().numpy() if mask_kind == 2 else None)
        assert_close(z[s].float().cpu().numpy(), ref, f"sequence {b} of {batch}x{seq} m{mask_kind}")

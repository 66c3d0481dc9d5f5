"""Dense Linear + residual + LayerNorm on persistent clusters of CTA pairs: remainders of the 256-row
blocks, one to several blocks per cluster, every width, K below one block and with a remainder, against
plain fp32 math, and its use by a whole encoder layer."""
import ctypes

import numpy as np
import pytest

from conftest import assert_close

pytestmark = pytest.mark.gpu


@pytest.fixture
def pair_ln(et):
    def force(mode):
        et.lib().et_debug_set_pair_ln(ctypes.c_int(mode), ctypes.c_int(768))
    yield force
    force(-1)


@pytest.mark.parametrize("T,K,N", [
    (1, 64, 512), (33, 16, 768), (255, 80, 1024), (256, 768, 768), (257, 1040, 768),
    (6145, 256, 768), (6400, 144, 512), (12805, 64, 1024), (20000, 512, 512),
])
@pytest.mark.parametrize("bias", [True, False])
def test_linear_skip_layernorm_pairs(et, cuda, pair_ln, T, K, N, bias):
    import torch
    g = torch.Generator(device=cuda)
    g.manual_seed(T + K + N)
    rand = lambda *s, std=1.0: (torch.randn(s, generator=g, device=cuda) * std).half()
    x, w, r = rand(T, K), rand(N, K, std=K ** -0.5), rand(T, N)
    b = rand(N) if bias else None
    gamma, beta = rand(N) + 1.0, rand(N)
    pair_ln(1)
    out = torch.full((T, N), float("nan"), dtype=torch.float16, device=cuda)
    et.linear_skip_layernorm(x, w, b, r, gamma, beta, out=out)
    assert et.device_error() == 0
    v = x.float() @ w.float().t() + (b.float() if bias else 0.0) + r.float()
    ref = torch.nn.functional.layer_norm(v, (N,), gamma.float(), beta.float(), 1e-5)
    # one fp16 rounding of values of size |gamma| * 4 or so, fp32 everything before it
    assert_close(out.float().cpu().numpy(), ref.cpu().numpy(), f"T{T} K{K} N{N}", rel_tol=1e-3)
    again = et.linear_skip_layernorm(x, w, b, r, gamma, beta)
    assert torch.equal(out, again)


def test_encoder_layer_with_pair_ln(et, cuda, pair_ln):
    """One layer of 4200 tokens: the pair form against the separate GEMM and LayerNorm."""
    import torch
    batch, seq, hidden, heads, ff = 12, 350, 768, 12, 3072
    g = torch.Generator(device=cuda)
    g.manual_seed(5)
    rand = lambda *s, std=0.02: (torch.randn(s, generator=g, device=cuda) * std).half().cpu().numpy()
    w = {"wqkv": rand(3 * hidden, hidden), "bqkv": rand(3 * hidden), "wo": rand(hidden, hidden),
         "bo": rand(hidden), "w1": rand(ff, hidden), "b1": rand(ff), "w2": rand(hidden, ff), "b2": rand(hidden)}
    for ln in ("ln1", "ln2"):
        w[ln + "_g"] = np.ones(hidden, np.float16)
        w[ln + "_b"] = np.zeros(hidden, np.float16)
    stack = et.EncoderStack([et.EncoderLayer(w, heads, et.ACT_GELU)], batch, seq)
    x = torch.randn((batch * seq, hidden), generator=g, device=cuda).half()
    outs = []
    for mode in (0, 1):
        pair_ln(mode)
        outs.append(stack.forward(x).float().cpu().numpy())
        assert et.device_error() == 0
    # the separate pass rounds the product to fp16 before the LayerNorm: 2^-11 relative, twice a layer
    assert_close(outs[1], outs[0], "pair LayerNorm layer", rel_tol=1.5e-3)

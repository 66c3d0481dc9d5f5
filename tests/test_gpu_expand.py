"""GPU parity of the Linear layers whose weights are expanded to operand tiles in shared memory
(1x16 vectors, CSR, packed tiles) at the edges of their tiling: partial token blocks, several
token blocks per CTA, partial feature panels of every width, K not a multiple of a block, weight
buffers that wrap, empty and full weights; CSR rows in any order and with repeated columns.

Tolerance: both sides accumulate fp16 products in fp32, so they differ by the rounding of the fp16
output, at most 2^-11 of the largest |y|, plus fp32 summation order (K * 2^-24 of sum |w x|, far
below it).  GELU adds the 5e-4 absolute error of tanh.approx."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [
    # T, in, out
    (1, 16, 16), (128, 768, 768), (129, 80, 144), (300, 1024, 48), (700, 1040, 3088), (2048, 256, 2304),
    (4100, 192, 1008), (64, 3072, 768),
]


def _dev(a, cuda):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).to(cuda)


def _check(y, ref, what):
    y = y.float().cpu().numpy()
    tol = 2.0 ** -11 * np.abs(ref).max() + 6e-4
    assert np.isfinite(y).all() and np.abs(y - ref).max() <= tol, f"{what}: {np.abs(y - ref).max()} > {tol}"


def _case(et, seed, T, inn, out):
    return (et.synth.normal_fast(seed, 1, (T, inn), 1.0), et.synth.normal_fast(seed, 2, (out, inn), 0.05),
            et.synth.normal_fast(seed, 3, (out,), 0.1))


@pytest.mark.parametrize("sparsity", [0.0, 0.9, 1.0])
@pytest.mark.parametrize("T,inn,out", SHAPES)
def test_1x16(et, orc, cuda, T, inn, out, sparsity):
    x, w, b = _case(et, 71, T, inn, out)
    w = et.synth.prune_1x16(w, 71, 6, sparsity)
    ti, ri, data = et.synth.dense_to_1x16(w)
    n = len(ri)
    y = et.linear_1x16(_dev(x, cuda), _dev(ti, cuda), _dev(ri, cuda) if n else None,
                       _dev(data, cuda) if n else None, out, _dev(b, cuda), 2)
    assert et.device_error() == 0
    _check(y, orc.linear_dense(x, w, b, 2), f"1x16 {T}x{inn}x{out} s={sparsity}")


@pytest.mark.parametrize("sparsity", [0.5, 0.97])
@pytest.mark.parametrize("T,inn,out", SHAPES + [(130, 8192, 40), (77, 1000, 203), (260, 24, 5)])
def test_csr(et, orc, cuda, T, inn, out, sparsity):
    x, w, b = _case(et, 72, T, inn, out)
    w = w * (et.synth.uniform(72, 7, out * inn).reshape(out, inn) >= sparsity)
    ip, ix, data = et.synth.dense_to_csr(w)
    n = len(ix)
    y = et.linear_csr(_dev(x, cuda), _dev(ip, cuda), _dev(ix, cuda) if n else None,
                      _dev(data, cuda) if n else None, out, _dev(b, cuda), 1)
    assert et.device_error() == 0
    _check(y, orc.linear_dense(x, w, b, 1), f"csr {T}x{inn}x{out} s={sparsity}")


@pytest.mark.parametrize("inn", [256, 3072])
def test_csr_rows_in_any_order_and_repeated_columns(et, orc, cuda, inn):
    T, out = 200, 100
    x, w, b = _case(et, 73, T, inn, out)
    rng = np.random.default_rng(5)
    ip, ix, data = [0], [], []
    for r in range(out):
        cols = rng.permutation(inn)[:20]
        if r % 7 == 3:
            cols[5] = cols[11]  # one column twice: its values add up
        ix += list(cols)
        data += list(w[r, rng.permutation(inn)[:20]])
        ip.append(len(ix))
    ip, ix, data = np.array(ip, np.int32), np.array(ix, np.int32), np.array(data, np.float16)
    y = et.linear_csr(_dev(x, cuda), _dev(ip, cuda), _dev(ix, cuda), _dev(data, cuda), out, _dev(b, cuda), 0)
    assert et.device_error() == 0
    _check(y, orc.linear_csr(x, ip, ix, data, out, b, 0), f"unordered csr, in {inn}")


@pytest.mark.parametrize("sparsity", [0.0, 0.8, 0.95])
@pytest.mark.parametrize("T,inn,out", SHAPES)
def test_packed_tiles(et, orc, cuda, T, inn, out, sparsity):
    import ctypes
    import torch
    x, w, b = _case(et, 74, T, inn, out)
    w = et.synth.prune_tiles(w, 74, 4, sparsity)
    rp, ro, tiles = et.synth.dense_to_tile(w)
    pk = et.PackedTiles(rp, ro, tiles, inn, out, cuda)
    L = et.lib()
    ys = []
    for mode in (2, 0):  # expanded tiles; one tensor-core product per stored tile
        L.et_debug_set_tile_persist(ctypes.c_int(mode))
        try:
            ys.append(et.linear_tile_packed(_dev(x, cuda), pk, _dev(b, cuda), 2))
            assert et.device_error() == 0
        finally:
            L.et_debug_set_tile_persist(ctypes.c_int(-1))
    _check(ys[0], orc.linear_dense(x, w, b, 2), f"packed {T}x{inn}x{out} s={sparsity}")
    # on finite activations the products of absent tiles add exact zeros: the same bits
    assert torch.equal(ys[0], ys[1])


def _with_infinities(et, seed, T, inn):
    """Activations with infinities of both signs and NaN in a few (token, feature) places."""
    x = et.synth.normal_fast(seed, 1, (T, inn), 1.0)
    for i, t in enumerate(range(0, T, 3)):
        x[t, (37 * i + 5) % inn] = (np.inf, -np.inf, np.nan, 65504.0)[i % 4]
        if i % 5 == 0:
            x[t, (11 * i) % inn] = np.inf
    return x


def _same_with_infinities(y, ref, what):
    y, ref = y.float().cpu().numpy(), ref.astype(np.float32)
    assert np.array_equal(np.isnan(y), np.isnan(ref)), f"{what}: NaN in other places"
    inf = np.isinf(ref)
    assert np.array_equal(np.isinf(y), inf) and np.array_equal(y[inf], ref[inf]), f"{what}: infinities"
    fin = np.isfinite(ref)
    # the fp16 rounding of the output and, per token, fp32 sums of terms as large as 65504 * |w|
    scale = np.abs(np.where(fin, ref, 0)).max(axis=1, keepdims=True)
    d = np.abs(np.where(fin, y, 0) - np.where(fin, ref, 0))
    assert (d <= 2.0 ** -10 * scale + 6e-4).all(), f"{what}: {d.max()}"


@pytest.mark.parametrize("T,inn,out", [(40, 256, 48), (200, 2048, 112), (1100, 768, 272)])
def test_an_infinity_reaches_only_outputs_that_store_a_weight_for_it(et, orc, cuda, T, inn, out):
    """Expanded operands hold zeros where nothing is stored, and 0 * inf is NaN: the product must still be the
    sum over stored entries, whichever kernel the token count selects for packed tiles."""
    import ctypes
    x = _with_infinities(et, 75, T, inn)
    xf, b = x.astype(np.float32), et.synth.normal_fast(75, 3, (out,), 0.1)
    w = et.synth.normal_fast(75, 2, (out, inn), 0.05)
    d = lambda a: _dev(a, cuda)
    with np.errstate(invalid="ignore"):
        wv = et.synth.prune_1x16(w, 75, 6, 0.8)
        ti, ri, dv = et.synth.dense_to_1x16(wv)
        y = et.linear_1x16(d(x), d(ti), d(ri), d(dv), out, d(b), 0)
        _same_with_infinities(y, orc.linear_1x16(xf, ti, ri, dv, out, b, 0), "1x16")
        wc = w * (et.synth.uniform(75, 7, out * inn).reshape(out, inn) >= 0.9)
        ip, ix, dc = et.synth.dense_to_csr(wc)
        for mode in (0, 1):  # expanded, by stored values
            et.lib().et_debug_set_csr_rows(ctypes.c_int(mode))
            try:
                y = et.linear_csr(d(x), d(ip), d(ix), d(dc), out, d(b), 0)
            finally:
                et.lib().et_debug_set_csr_rows(ctypes.c_int(-1))
            _same_with_infinities(y, orc.linear_csr(xf, ip, ix, dc, out, b, 0), f"csr {mode}")
        wt = et.synth.prune_tiles(w, 75, 4, 0.8)
        rp, ro, tiles = et.synth.dense_to_tile(wt)
        ref = orc.linear_tile(xf, rp, ro, tiles, out, b, 0)
        pk = et.PackedTiles(rp, ro, tiles, inn, out, cuda)
        for mode in (-1, 2, 0):  # automatic, expanded tiles, one product per stored tile
            et.lib().et_debug_set_tile_persist(ctypes.c_int(mode))
            try:
                y = et.linear_tile_packed(d(x), pk, d(b), 0)
            finally:
                et.lib().et_debug_set_tile_persist(ctypes.c_int(-1))
            _same_with_infinities(y, ref, f"packed tiles, mode {mode}")
    assert et.device_error() == 0


def test_first_calls_of_narrow_and_wide_layers_from_many_threads(et, cuda):
    """The kernel's shared-memory limit belongs to the process: whichever thread's first call comes last, wide
    layers (192 KB) must still launch beside narrow ones."""
    import subprocess
    import sys
    from conftest import ROOT
    code = """
import importlib, sys, threading
sys.path.insert(0, %r)
import torch
et = importlib.import_module("scpaper-2021_b200")
def layer(inn):
    out = 64
    ip = torch.arange(out + 1, dtype=torch.int32, device="cuda") * 400
    ix = torch.arange(400, dtype=torch.int32, device="cuda").repeat(out)
    return (torch.ones(8, inn, device="cuda").half(), ip, ix, torch.ones(400 * out, device="cuda").half(), out)
layers = [layer(i) for i in (8192, 512, 1024, 4096) * 4]
et.lib()
start, bad = threading.Barrier(len(layers)), []
def work(a):
    start.wait()
    try:
        for _ in range(20):
            et.linear_csr(*a)
    except Exception as e:
        bad.append(e)
ts = [threading.Thread(target=work, args=(a,)) for a in layers]
[t.start() for t in ts]; [t.join() for t in ts]
y = et.linear_csr(*layers[0])
torch.cuda.synchronize()
assert not bad, bad
assert (y == 400).all() and et.device_error() == 0
""" % ROOT
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=180)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("T,inn,out,sparsity", [(1, 16, 16, 0.9), (9, 24, 5, 0.5), (77, 1000, 203, 0.97),
                                                (130, 8192, 40, 0.999), (300, 1024, 515, 1.0)])
def test_csr_by_stored_values(et, orc, cuda, T, inn, out, sparsity):
    """The kernel for almost empty weights, at its remainders (8 tokens, 256 features) and its widest row."""
    import ctypes
    x, w, b = _case(et, 78, T, inn, out)
    w = w * (et.synth.uniform(78, 7, out * inn).reshape(out, inn) >= sparsity)
    ip, ix, data = et.synth.dense_to_csr(w)
    n = len(ix)
    ref = orc.linear_csr(x, ip, ix, data, out, b, 1)
    for mode in (1, 0, -1):
        et.lib().et_debug_set_csr_rows(ctypes.c_int(mode))
        try:
            y = et.linear_csr(_dev(x, cuda), _dev(ip, cuda), _dev(ix, cuda) if n else None,
                              _dev(data, cuda) if n else None, out, _dev(b, cuda), 1)
        finally:
            et.lib().et_debug_set_csr_rows(ctypes.c_int(-1))
        assert et.device_error() == 0
        _check(y, ref, f"csr by values {T}x{inn}x{out} mode {mode}")

"""Runs the C++ driver that exercises the reference-compatible host classes
(scpaper-2021_b200/host/: Linear<MAT>, Attention<config>, Encoder<config>, ...) on the GPU."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BIN = os.path.join(ROOT, "tests", "cpp", "host_api_test.bin")


@pytest.mark.gpu
def test_cpp_host_api(cuda, orc):
    if not os.path.exists(BIN):
        import __graft_entry__ as entry
        entry.build_cpp_tests()
    r = subprocess.run([BIN], capture_output=True, text=True, timeout=600)
    print(r.stdout[-4000:])
    print(r.stderr[-2000:])
    assert r.returncode == 0, r.stdout[-3000:]
    assert "all host-API checks passed" in r.stdout


def test_first_calls_of_a_fresh_thread(et, cuda):
    """A host thread that has not touched the device yet has no context of its own: the first call it makes may
    be any operator."""
    import threading

    import torch
    x, w = torch.ones((8, 512), device=cuda).half(), torch.ones((64, 512), device=cuda).half()
    ip = torch.arange(65, dtype=torch.int32, device=cuda) * 400
    ix = torch.arange(400, dtype=torch.int32, device=cuda).repeat(64)
    data, y = torch.ones(25600, device=cuda).half(), torch.empty((8, 64), device=cuda).half()
    ti = torch.zeros((4, 33), dtype=torch.int32, device=cuda)
    torch.cuda.synchronize()
    failed = []

    def first(name, call):
        def go():
            try:
                call()
            except et.EtError as e:
                failed.append((name, str(e)))
        t = threading.Thread(target=go)
        t.start()
        t.join()

    first("csr", lambda: et.linear_csr(x, ip, ix, data, 64))
    first("1x16", lambda: et.linear_1x16(x, ti, None, None, 64))
    first("dense", lambda: et.linear_dense(x, w, out=y))
    torch.cuda.synchronize()
    assert not failed and et.device_error() == 0, failed
    assert (y == 512).all()

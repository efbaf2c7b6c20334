"""A matrix assembled again: other ranks in the same device arrays, products in flight on a user's
stream, and another thread that captures a stream meanwhile."""
import threading

import numpy as np
import pytest
from conftest import rel

pytestmark = pytest.mark.gpu


def _matrix(hb, vt=1, n=3000, eps=1e-4, ell=0.3, assemble=True):
    pts = np.random.default_rng(n).random((n, 3))
    hb.set_parameters(compressionMinLeafSize=0)
    return hb.HMatrix(pts, hb.kernel(hb.EXP_COV, ell=ell, nugget=1e-6), value_type=vt, leaf_size=64, eta=2.0,
                      epsilon=eps, assemble=assemble)


def test_assembly_while_another_thread_captures(hb):
    import torch
    h = _matrix(hb, assemble=False)
    try:
        y = torch.zeros(1000, device="cuda")
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        errors = []

        def assemble():
            try:
                h.assemble()
                h.assemble()
            except Exception as e:  # noqa: BLE001  (reported by the asserts below)
                errors.append(e)

        torch.cuda.synchronize()
        t = threading.Thread(target=assemble)
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            y.add_(1.0)
            t.start()
            t.join()
            y.add_(1.0)
        assert not errors, errors
        graph.replay()
        torch.cuda.synchronize()
        assert torch.all(y == 2.0)
        x = np.random.default_rng(0).standard_normal((h.n, 1))
        fresh = _matrix(hb)
        assert rel(h.gemv(x), fresh.gemv(x)) < 1e-13
        fresh.close()
    finally:
        h.close()


@pytest.mark.parametrize("vt", [0, 1])
def test_other_ranks_with_products_in_flight(hb, vt):
    """Looser, tighter, looser and much smaller ranks on one handle: each time the products queued
    before the assembly are those of the old matrix, and the new one equals a matrix built afresh."""
    import torch
    h = _matrix(hb, vt, eps=1e-4)
    dt = torch.float64 if vt == 1 else torch.float32
    tol = 1e-13 if vt == 1 else 1e-6
    stream = torch.cuda.Stream()
    try:
        g = np.random.default_rng(1)
        x = torch.from_numpy(np.ascontiguousarray(g.standard_normal((5, h.n)))).to("cuda", dt)
        for eps in (1e-7, 1e-4, 1e-1, 1e-6):
            want = {}
            for trans in "NT":
                y = torch.empty_like(x)
                h.gemv_device(x.data_ptr(), y.data_ptr(), 5, trans=trans, stream=stream.cuda_stream)
                stream.synchronize()
                want[trans] = y
            got = {t: torch.empty_like(x) for t in "NT"}
            torch.cuda.synchronize()
            with torch.cuda.stream(stream):
                torch.cuda._sleep(200_000_000)  # about a tenth of a second: the products queue behind it
            for trans in "NT":
                for _ in range(10):
                    h.gemv_device(x.data_ptr(), got[trans].data_ptr(), 5, trans=trans, stream=stream.cuda_stream)
            h.set_low_rank_epsilon(eps)
            h.lib.hmat_delete_compression(h._comp)
            h._comp = h.lib.hmat_create_compression_aca_plus(eps)
            h.assemble()
            stream.synchronize()
            for trans in "NT":
                assert torch.equal(got[trans], want[trans]), (eps, trans)
            fresh = _matrix(hb, vt, eps=eps)
            try:
                assert np.array_equal(h.leaf_table(), fresh.leaf_table())
                for trans in "NT":
                    a, b = torch.empty_like(x), torch.empty_like(x)
                    h.gemv_device(x.data_ptr(), a.data_ptr(), 5, trans=trans)
                    fresh.gemv_device(x.data_ptr(), b.data_ptr(), 5, trans=trans)
                    torch.cuda.synchronize()
                    assert rel(a.cpu().numpy(), b.cpu().numpy()) <= tol
            finally:
                fresh.close()
    finally:
        h.close()


NO_THREADS = r"""
import ctypes, sys
sys.path.insert(0, "tests")
import conftest
import numpy as np
hb = conftest.load_engine_package()
hb.set_parameters(compressionMinLeafSize=0)
pts = np.random.default_rng(0).random((8000, 3))
h = hb.HMatrix(pts, hb.kernel(hb.EXP_COV, ell=0.3, nugget=1e-6), leaf_size=64, eta=2.0, epsilon=1e-4)
assert h.payload_layout()[1] > 4 << 20  # large enough to be planned on two threads
x = np.random.default_rng(1).standard_normal((8000, 2))
want = h.gemv(x), h.gemv(x, trans="T")
libc = ctypes.CDLL(None)
attr = ctypes.create_string_buffer(256)
assert libc.pthread_attr_init(attr) == 0
assert libc.pthread_attr_setstacksize(attr, ctypes.c_size_t(1 << 47)) == 0
assert libc.pthread_setattr_default_np(attr) == 0  # no further thread can be started: its stack cannot be mapped
h.assemble()
got = h.gemv(x), h.gemv(x, trans="T")
assert all(np.array_equal(a, b) for a, b in zip(got, want))
h.close()
print("assembled")
"""


def test_assembly_where_no_thread_can_be_started():
    import subprocess
    import sys

    from conftest import ROOT
    r = subprocess.run([sys.executable, "-c", NO_THREADS], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "assembled" in r.stdout, r.stderr[-2000:]

"""Device memory that CSR builds and community listings keep between calls:
bounded, and given back when an engine ends, when one of the library's
allocations fails, and on request; a device context that ends afterwards
leaves nothing behind that a later call would use."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

import lvb200
from conftest import PKG

pytestmark = pytest.mark.gpu

N, M = 100_000, 6_000_000
SCRATCH = 4 * 2 * M * 4  # keys, columns and weights of the 2 M entries, once more each


def _free():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _build(src, dst, off, col, w):
    nnz = ctypes.c_uint64()
    assert lvb200.lib().lv_csr_from_edges_device(N, M, src.data_ptr(), dst.data_ptr(), None,
                                                 off.data_ptr(), col.data_ptr(), w.data_ptr(),
                                                 ctypes.byref(nnz), None) == 0


@pytest.mark.parametrize("how", ["engine_ends", "allocation_fails", "request"])
def test_scratch_is_given_back(how):
    import torch

    src = torch.randint(0, N, (M,), dtype=torch.int32, device="cuda")
    dst = torch.randint(0, N, (M,), dtype=torch.int32, device="cuda")
    out = (torch.empty(N + 1, dtype=torch.int64, device="cuda"),
           torch.empty(2 * M, dtype=torch.int32, device="cuda"),
           torch.empty(2 * M, dtype=torch.float32, device="cuda"))
    small = lvb200.Graph.from_edges(3, [0, 1], [1, 2])
    _build(src, dst, *out)
    lvb200.Engine().close()  # gives back what calls before kept
    with lvb200.Engine() as e:
        base = _free()
        _build(src, dst, *out)
        kept = base - _free()
        assert SCRATCH // 2 < kept <= 512 << 20
        if how == "allocation_fails":
            lvb200.fail_device_alloc(1)
            try:
                with pytest.raises(lvb200.LouvainError):
                    e.load(small)
            finally:
                lvb200.fail_device_alloc(0)
        elif how == "request":
            lvb200.release_scratch(0)
        else:
            lvb200.Engine().close()
        assert base - _free() < SCRATCH // 8
        _build(src, dst, *out)  # and the next call finds its scratch


SCRIPT = r"""
import ctypes
import numpy as np
import lvb200

rt = ctypes.CDLL("libcudart.so.12")
rng = np.random.default_rng(1)
n, m = 1000, 50_000
src, dst = rng.integers(0, n, m).astype(np.uint32), rng.integers(0, n, m).astype(np.uint32)

def malloc(size):
    p = ctypes.c_void_p()
    assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(size)) == 0
    return p

def device(a):
    p = malloc(a.nbytes)
    assert rt.cudaMemcpy(p, a.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(a.nbytes), 1) == 0
    return p

def with_engine():
    with lvb200.Engine() as e:
        e.load_edges(n, src, dst)
        while e.phase_move(1e-6)[0]:
            e.phase_aggregate()
        return [np.array(x) for x in e.communities()]

def without():
    off = malloc(8 * (n + 1))
    nnz = ctypes.c_uint64()
    assert lvb200.lib().lv_csr_from_edges_device(n, m, device(src), device(dst), None, off,
                                                 malloc(8 * m), malloc(8 * m),
                                                 ctypes.byref(nnz), None) == 0
    out = np.zeros(n + 1, np.uint64)
    assert rt.cudaMemcpy(out.ctypes.data_as(ctypes.c_void_p), off, ctypes.c_size_t(out.nbytes),
                         2) == 0
    return [out]

for f, end in ((with_engine, lambda: None), (without, lvb200.release_scratch)):
    a = f()
    end()
    assert rt.cudaDeviceReset() == 0
    b = f()
    end()
    assert all(np.array_equal(x, y) for x, y in zip(a, b))
    assert rt.cudaDeviceReset() == 0
print("same")
"""


def test_sorts_in_a_new_context():
    env = dict(os.environ, PYTHONPATH=os.path.join(PKG, "python"))
    r = subprocess.run([sys.executable, "-c", SCRIPT], env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stderr[-2000:]

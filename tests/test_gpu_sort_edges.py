"""The radix passes behind the device CSR build and the community listing at
the sizes where a pass can go wrong: entry counts around a tile (4096
entries), key widths around a digit boundary (one to four passes), pointers
that are not 16-byte aligned, self-loops, and one community or row only.
The host reader and a host grouping are the reference; every value is
equal."""
import ctypes

import numpy as np
import pytest

import lvb200

pytestmark = pytest.mark.gpu


def _edges(n, m, seed):
    rng = np.random.default_rng(seed)
    src = (n * rng.random(m) ** 2).astype(np.uint32)
    dst = rng.integers(0, n, m).astype(np.uint32)
    dst[: m // 7] = src[: m // 7]
    return src, dst, rng.normal(size=m).astype(np.float32)


@pytest.mark.parametrize("n", [1, 2, 255, 256, 65_537, (1 << 24) + 3])
@pytest.mark.parametrize("m", [1, 2047, 2048, 2049, 30_001])
@pytest.mark.parametrize("shift", [0, 1])
def test_device_csr_at_tile_and_digit_edges(n, m, shift):
    import torch

    src, dst, w = _edges(n, m, seed=n % 1000 + m)
    want_n, off, col, ww, _ = lvb200.Graph.from_edges(n, src, dst, w).csr()

    def dev(a):  # `shift` elements past an allocation's start
        t = torch.zeros(m + shift, dtype=torch.int32, device="cuda")
        t[shift:] = torch.from_numpy(a.view(np.int32))
        return t[shift:]

    d_src, d_dst, d_w = dev(src), dev(dst), dev(w)
    d_off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    d_col = torch.zeros(2 * m, dtype=torch.int32, device="cuda")
    d_out = torch.zeros(2 * m, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    nnz = ctypes.c_uint64()
    assert lvb200.lib().lv_csr_from_edges_device(
        n, m, d_src.data_ptr(), d_dst.data_ptr(), d_w.data_ptr(), d_off.data_ptr(),
        d_col.data_ptr(), d_out.data_ptr(), ctypes.byref(nnz), None) == 0
    e = nnz.value
    assert want_n == n and e == len(col)
    assert np.array_equal(d_off.cpu().numpy().view(np.uint64), off)
    assert np.array_equal(d_col[:e].cpu().numpy().view(np.uint32), col)
    assert np.array_equal(d_out[:e].cpu().numpy(), ww)


@pytest.mark.parametrize("n,comms", [(1, 1), (4096, 1), (4097, 4097), (10_000, 257), (70_000, 70_000)])
def test_listing_at_digit_edges(n, comms):
    # isolated vertices, one ring per community: the partition is known
    comm = np.sort(np.random.default_rng(n).integers(0, comms, n).astype(np.uint32))
    comm = np.unique(comm, return_inverse=True)[1].astype(np.uint32)
    order = np.argsort(comm, kind="stable")
    with lvb200.Engine() as e:
        e.load(lvb200.Graph.from_csr(n, np.zeros(n + 1, np.uint64), [], []))
        e.set_level_comm(order[np.searchsorted(comm[order], comm)].astype(np.uint32))
        part = e.assignment()
        offsets, members = e.communities()
    assert len(offsets) == n + 1  # ids below the level's vertex count
    want = np.argsort(part, kind="stable")
    assert np.array_equal(members, want.astype(np.uint32))
    assert np.array_equal(offsets, np.searchsorted(part[want], np.arange(n + 1)))

"""The allocation-free sum at its edges: remainders of the 4-element vectors, buffers that are only
4-byte aligned, the smallest and largest size, every number of buffers."""

import ctypes

import pytest
import torch

from test_zz_no_alloc import _call, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1])  # elements from a 16-byte boundary
@pytest.mark.parametrize("n", [1, 3, 4, 511, 512, 513, 4095])
@pytest.mark.parametrize("world", [2, 3, 5, 8])
def test_sum_in_buffer_order(world, n, offset):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    gen = torch.Generator().manual_seed(17 * n + world)
    pads = [torch.randn(n + 8, generator=gen).cuda() for _ in range(world)]
    before = [p.clone() for p in pads]
    expect = before[0][offset:offset + n].clone()
    for p in before[1:]:
        expect += p[offset:offset + n]  # the same fp32 additions in the same order: bit for bit
    rc, msg = _call(_lib(), [p[offset:offset + n] for p in pads])
    assert rc == 0, msg
    for p, b in zip(pads, before):
        assert torch.equal(p[offset:offset + n], expect)
        assert torch.equal(p[:offset], b[:offset]) and torch.equal(p[offset + n:], b[offset + n:])


def test_an_error_that_the_host_has_pending():
    """It is neither reported by this call nor cleared."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    bufs = [torch.full((9,), float(r), device="cuda") for r in range(3)]
    torch.cuda.synchronize()
    runtime = ctypes.CDLL("libcudart.so.12")  # the one that torch and the library use
    refused = runtime.cudaSetDevice(4096)  # no such device: an error of the host call alone
    assert refused != 0
    rc, msg = _call(_lib(), bufs)
    assert runtime.cudaGetLastError() == refused
    assert rc == 0, msg
    assert all(bool((b == 3.0).all()) for b in bufs)

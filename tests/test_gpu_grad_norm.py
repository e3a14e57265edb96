"""Sum of squares and gradient norm at the edges of their vectors, batches and blocks, against fp64."""

import pytest
import torch

pytestmark = pytest.mark.gpu


# no element, remainders of a vector, one block and one more vector, several batches of the whole grid
@pytest.mark.parametrize("n", [0, 1, 3, 4, 5, 2047, 2048, 2052, 300_001, 5_000_003])
def test_sum_of_squares(n):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from fairring_b200 import _C
    from fairring_b200.ops import FlatAdamW

    x = torch.randn(n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n))
    want = float(x.double().pow(2).sum())
    # an fp32 sum of up to n / 300000 + 32 terms per thread, then fp64
    assert abs(float(_C.sumsq(x)) - want) <= 1e-5 * want
    norm = FlatAdamW(torch.zeros_like(x), x).grad_norm()
    assert norm.shape == (1,) and abs(float(norm) - want ** 0.5) <= 1e-5 * want ** 0.5
    assert torch.equal(norm, FlatAdamW(torch.zeros_like(x), x).grad_norm())  # always in the same order

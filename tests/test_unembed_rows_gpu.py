"""Un-embedding of 9 to 64 rows: the register-tiled kernel's running sums against 64 bits."""
import math

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("k", [36, 256, 260, 1600, 6144])
def test_error_does_not_grow_with_a_long_chain_of_roundings(rows, k):
    """A sum of n random terms, one after the other, ends about 0.4 u sqrt(n / 2) of its size away from the exact one (u = 2^-24: the partial sums grow
    like sqrt(i), each rounded to half a unit at most).  Here n is at most 128 pairs in a run, then k / 256 runs; the bound allows 0.5 u sqrt(n) for both and
    u for the products.  One chain over all of k = 6144 would be at 0.4 u sqrt(1536) = 9e-7, the bound is 5.4e-7."""
    import torch
    import gpt_b200
    n = 20000      # 157 column tiles: k is not shared by a cluster
    gen = torch.Generator(device="cuda").manual_seed(rows * k)
    x = torch.randn(rows, k, device="cuda", generator=gen)
    w = torch.randn(n, k, device="cuda", generator=gen) * 0.02
    y = torch.full((rows, n), float("nan"), device="cuda")
    b = gpt_b200.Backend(0)
    b.device_unembedding_forward(y, x, w, 1, rows, k, n)
    b.synchronize()
    b.close()
    want = x.double() @ w.double().t()
    error = float((y.double() - want).norm() / want.norm())
    assert error <= 2.0 ** -24 * (0.5 * math.sqrt(min(k / 2, 128)) + 0.5 * math.sqrt(k / 256) + 1.0), error

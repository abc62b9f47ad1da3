"""The kernels that a rule on sizes or alignment chooses, at the edges of their tiles, against the general kernel of
the same operation (bit for bit where the sums have the same order) or a float64 reference."""

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
EPS = 2.0 ** -24  # half a unit in the last place of float32


@pytest.fixture(scope="module")
def ops32():
    from fastgen_b200.csrc.ops import Ops
    return Ops(torch.float32, DEV)


@pytest.fixture(scope="module")
def ops16():
    from fastgen_b200.csrc.ops import Ops
    return Ops(torch.bfloat16, DEV)


def _randn(gen, *shape, scale=1.0):
    return (torch.randn(*shape, generator=gen) * scale).to(DEV)


# -- the float32 product ----------------------------------------------------------------------------

@pytest.mark.parametrize("m,n,k", [
    (1, 16, 4), (7, 17, 132), (8, 2051, 128), (8, 40, 1028),           # few rows, a row a lane
    (9, 33, 100), (31, 200, 2048), (33, 5120, 36), (64, 15, 260),      # few rows, four a lane
    (9, 5200, 36), (24, 5300, 68), (32, 9001, 32),                     # small blocks of 1 to 4 warps
    (65, 64, 4), (97, 65, 100), (160, 2047, 64), (321, 63, 33 * 4),    # small blocks
    (64, 9000, 36), (65, 7001, 32), (200, 5121, 40), (777, 2050, 28),  # 128 columns by 3 to 8 warps
    (33, 37889, 16), (65, 19201, 20), (777, 3100, 36),                 # 64 x 128 tiles
])
def test_float32_product_routes(ops32, m, n, k):
    """Every kernel gives the bits of the general one (taken for rows that are no multiple of 16 bytes)."""
    g = torch.Generator().manual_seed(m * 7 + n)
    x, w, bias = _randn(g, m, k), _randn(g, n, k), _randn(g, n)
    odd_x, odd_w = torch.empty(m, k + 1, device=DEV)[:, :k], torch.empty(n, k + 3, device=DEV)[:, :k]
    odd_x.copy_(x)
    odd_w.copy_(w)
    got, want = ops32.linear(x, w), ops32.linear(odd_x, odd_w)
    assert torch.equal(got, want)
    assert torch.equal(ops32.linear(x, w, bias=bias), ops32.linear(odd_x, odd_w, bias=bias))
    wide = torch.full((m, n + 5), 3.0, device=DEV)  # rows of the result that are no multiple of 16 bytes
    ops32.linear(x, w, out=wide[:, :n])
    assert torch.equal(wide[:, :n], want) and bool((wide[:, n:] == 3.0).all())
    ref = x.double() @ w.double().T
    bound = k * EPS * (x.double().abs() @ w.double().abs().T)
    assert bool(((got.double() - ref).abs() <= bound + 1e-30).all())

"""Kernels that cut their rows into tiles, at the edges of the tiles."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def kernels():
    from kvcache_b200.kernels.api import CudaKernels
    return CudaKernels(DEV)


@pytest.mark.parametrize("N,K", [(1153, 132), (896, 4864), (9728, 100), (40, 77)])
def test_float32_product_rows_do_not_depend_on_the_tile(kernels, N, K):
    """Every number of rows at the edges of the tiles and of the rule that picks one: close to 64 bits, and each row bit for
    bit what it is in the largest step (one chain over k, whatever the tile)."""
    g = torch.Generator().manual_seed(31)
    x, w, bias = torch.randn(1001, K, generator=g), torch.randn(N, K, generator=g), torch.randn(N, generator=g)
    xd, wd, bd = x.to(DEV), w.to(DEV), bias.to(DEV)
    full = torch.empty(1001, N, device=DEV)
    kernels.linear(xd, wd, full, bd)
    # A chain of K rounded multiply-adds: at most K 2^-24 times the sum of magnitudes, which for normal numbers is 0.64 K.
    bound = K * 2.0 ** -24 * ((x.abs().double() @ w.abs().double().t()).max().item() + 5.0)
    assert (full.double().cpu() - (x.double() @ w.double().t() + bias.double())).abs().max().item() <= bound
    for M in (1, 4, 5, 16, 17, 48, 49, 64, 65, 129, 513):
        part = torch.full((M, N), float("nan"), device=DEV)
        kernels.linear(xd[:M], wd, part, bd)
        assert torch.equal(part, full[:M]), M

"""Routed products on tensor memory (csrc/gemm_grouped.cu): each width of tile that the number of row tiles and columns leads to, with
columns that end within a copied box and rows that end within a tile.  The router at the edges of its instances (csrc/moe.cu)."""
import pytest
import torch

from helpers import assert_close
from torch_kernels import TorchKernels

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SMS = 148


@pytest.fixture(scope="module")
def kernels():
    from kvcache_b200.kernels.api import CudaKernels
    return CudaKernels(DEV)


def _rand(*shape, seed, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(torch.bfloat16)


def _width(row_tiles, N, most):
    blocks = min(most * -(-N // 128), SMS)
    return min((256, 192, 128), key=lambda bn: -(-row_tiles * -(-N // bn) // blocks) * (128 + bn))     # the first of equals


@pytest.mark.parametrize("T,E,W,F,activation,widths", [(1030, 3, 48, 104, "swiglu", (128, 128)), (1100, 70, 336, 432, "relu2", (256, 192)),
                                                       (1100, 70, 200, 504, "clamped_swiglu", (256, 128)), (2300, 24, 1000, 1720, "relu2", (192, 192))])
def test_routed_products_of_every_width_of_tile(kernels, T, E, W, F, activation, widths):
    from kvcache_b200.engine.workspace import Workspace
    x = _rand(T, W, seed=1)
    N = F if activation == "relu2" else 2 * F
    w_up, w_down = _rand(E, N, W, seed=2, scale=0.1), _rand(E, W, F, seed=3, scale=0.1)
    chosen = torch.randint(0, E, (T, 1), generator=torch.Generator().manual_seed(4)).to(torch.int32)
    rows = torch.bincount(chosen.flatten(), minlength=E)
    row_tiles, most = int(((rows + 127) // 128).sum()), -(-T // 128) + E
    assert (_width(row_tiles, N, most), _width(row_tiles, W, most)) == widths
    share = torch.rand(T, 1, generator=torch.Generator().manual_seed(5))
    limit = 0.7 if activation == "clamped_swiglu" else 0.0
    ref, got = torch.zeros(T, W, dtype=torch.bfloat16), torch.full((T, W), 7.0, dtype=torch.bfloat16, device=DEV)
    TorchKernels(wide=True).routed_experts(x, w_up, w_down, chosen, share, ref, activation, limit=limit)
    kernels.routed_experts(x.to(DEV), w_up.to(DEV), w_down.to(DEV), chosen.to(DEV), share.to(DEV), got, activation, Workspace(DEV), limit=limit)
    kernels.check_errors()
    assert_close(got, ref, 2e-2)       # the activations and the products are rounded to 8 bits on the way, as in the other tests of it


@pytest.mark.parametrize("scores", ["chosen", "all"])
@pytest.mark.parametrize("E,top", [(1, 1), (32, 32), (33, 2), (128, 5), (129, 5), (1024, 3)])
def test_the_router_at_the_edges_of_its_instances(kernels, E, top, scores):
    logits = torch.randn(37, E, generator=torch.Generator().manual_seed(E))
    ref_c, ref_s = torch.zeros(37, top, dtype=torch.int32), torch.zeros(37, top)
    TorchKernels(wide=True).route_top(logits, ref_c, ref_s, scores=scores)
    got_c, got_s = torch.zeros(37, top, dtype=torch.int32, device=DEV), torch.zeros(37, top, device=DEV)
    kernels.route_top(logits.to(DEV), got_c, got_s, scores=scores)
    assert torch.equal(got_c.cpu(), ref_c)
    assert_close(got_s, ref_s, 1e-5)

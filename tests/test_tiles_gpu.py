"""Kernels that cut their rows into tiles, at the edges of the tiles."""
from __future__ import annotations

import dataclasses

import pytest
import torch

from helpers import assert_close, batch_to, clone_kv, paged_scenario
from torch_kernels import TorchKernels

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
REF = TorchKernels()


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


ROWS32 = [
    ([(0, 1), (63, 1), (64, 1), (500, 1)], 14, 2, 64, 64, 16, {}),                       # decoded tokens at the edge of a key tile
    ([(0, 65), (64, 64), (127, 3), (5, 1)], 6, 2, 64, 64, 16, {}),                       # tiles of rows that end inside a segment
    ([(700, 1), (3, 90), (0, 33)], 6, 2, 48, 80, 8, dict(window=100, keep_first=5)),     # kept keys beside a window; unequal sizes
    ([(700, 70), (3, 90)], 3, 1, 20, 4, 16, dict(chunk=48)),
    ([(0, 130), (900, 300)], 16, 2, 128, 128, 32, dict(window=64)),
    ([(200, 700)], 2, 2, 128, 100, 64, {}),
    ([(30, 1), (3, 2)], 2, 1, 16, 16, 16, {}),                                           # shared memory right below what needs no asking for
]


@pytest.mark.parametrize("scenario", ROWS32)
@pytest.mark.parametrize("options", [False, True])
def test_float32_attention_tiles(kernels, scenario, options):
    segments, Hq, Hkv, D, Dv, page, spec = scenario
    batch, kv = paged_scenario(segments, num_kv_heads=Hkv, head_dim=D, page_size=page, dtype=torch.float32, device="cpu", seed=41)
    g = torch.Generator().manual_seed(42)
    kv = dataclasses.replace(kv, v_pages=torch.randn(*kv.v_pages.shape[:3], Dv, generator=g),
                             spec=dataclasses.replace(kv.spec, value_dim=None if Dv == D else Dv, **spec))
    T = batch.num_tokens
    q = torch.randn(T, Hq * D, generator=g)
    more = dict(sink=torch.randn(Hq, generator=g), score_cap=5.0, slopes=torch.rand(Hq, generator=g) * 0.1) if options else {}
    ref = torch.empty(T, Hq * Dv)
    REF.paged_attention(q, batch, kv, ref, Hq, D ** -0.5, **more)
    there = {k: v.to(DEV) if torch.is_tensor(v) else v for k, v in more.items()}
    batch_dev, kv_dev = batch_to(batch, DEV), clone_kv(kv, DEV)
    # A later token's infinite value must not reach the rows before it: the last new token of every segment holds one.
    for i, (cached, new) in enumerate(segments):
        if new > 1:
            j = cached + new - 1
            kv_dev.v_pages[int(kv.block_table[i, j // page]), :, j % page] = float("inf")
    out = torch.empty(T, Hq * Dv, device=DEV)
    kernels.paged_attention(q.to(DEV), batch_dev, kv_dev, out, Hq, D ** -0.5, **there)
    kernels.check_errors()
    last = torch.tensor([sum(n for _, n in segments[:i + 1]) - 1 for i, (_, n) in enumerate(segments) if n > 1], dtype=torch.long)
    keep = torch.ones(T, dtype=torch.bool)
    keep[last] = False
    assert_close(out[keep.to(DEV)], ref[keep], 2e-6)
    # Each segment alone gives the same bits, whatever the tiles.
    at = 0
    for i, (cached, new) in enumerate(segments):
        alone, _ = paged_scenario([(cached, new)], num_kv_heads=Hkv, head_dim=D, page_size=page, dtype=torch.float32, device=DEV)
        one = torch.empty(new, Hq * Dv, device=DEV)
        kv_one = dataclasses.replace(kv_dev, block_table=kv_dev.block_table[i:i + 1].contiguous())
        kernels.paged_attention(q[at:at + new].to(DEV), alone, kv_one, one, Hq, D ** -0.5, **there)
        mine = slice(at, at + new - (1 if new > 1 else 0))
        assert torch.equal(one[:mine.stop - at], out[mine])
        at += new

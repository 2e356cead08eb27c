"""The two tensor-memory kernels for portions of prompts - pairs of row tiles against one line of work
(csrc/attention_pairs.cu), tiles cut into units by the host (csrc/attention_tc.cu) - on the same steps against float64."""
import dataclasses

import pytest
import torch

from helpers import assert_close, batch_to, clone_kv, paged_scenario
from torch_kernels import TorchKernels

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TOL = 1e-2                 # bfloat16 q, k, v, probabilities and results: 2^-9 each, as in the other tests of these kernels
REF = TorchKernels(wide=True)

# (segments (cached, new), Hq, Hkv, D, page, least key tiles of a block, window, kept first keys, chunk, sink, cap and slopes)
STEPS = [
    # a pair's rows around its tiles' edges: one row in the second tile, a full pair, one row in the next pair
    ([(0, 129)], 2, 1, 64, 16, 2, None, 0, None, False, False),
    ([(0, 127), (5, 128), (127, 256), (1, 257)], 3, 1, 128, 16, 2, None, 0, None, False, False),
    # at most 128 rows: two heads a stream, also of groups of odd size and of one
    ([(300, 128), (130, 2), (0, 100)], 7, 1, 64, 8, 1, None, 0, None, True, False),
    ([(900, 90), (255, 30)], 6, 2, 128, 64, 1, None, 0, None, False, True),
    ([(400, 77)], 2, 2, 128, 32, 1, None, 0, None, False, False),
    # streams cut over many blocks, blocks that take several pieces, pieces of one tile beside long ones
    ([(2500, 130), (0, 520)], 14, 2, 64, 16, 1, None, 0, None, False, False),
    ([(0, 1900)], 14, 2, 64, 16, 1, None, 0, None, False, False),
    ([(1300, 700), (0, 260), (64, 384)], 4, 2, 128, 16, 3, None, 0, None, True, False),
    # windows, kept first keys and chunks: places of the list that are no tile numbers, runs without any key
    ([(1500, 400), (20, 300)], 4, 1, 64, 16, 1, 200, 5, None, True, False),
    ([(2000, 300)], 4, 4, 128, 16, 1, 300, 400, None, False, False),
    ([(700, 600)], 6, 2, 64, 16, 2, 1, 0, None, False, False),
    ([(960, 500), (100, 280)], 4, 2, 128, 16, 1, None, 0, 192, False, False),
    # capped and biased scores
    ([(600, 300), (0, 150)], 6, 2, 64, 16, 1, None, 0, None, True, True),
]


@pytest.fixture(scope="module")
def kernels():
    from kvcache_b200.kernels.api import CudaKernels
    return CudaKernels(DEV)


@pytest.mark.parametrize("pairs", [True, False])
@pytest.mark.parametrize("step", STEPS)
def test_portions_through_both_tensor_memory_kernels(kernels, request, step, pairs):
    from kvcache_b200.engine.workspace import Workspace
    from kvcache_b200.parts.base import PagedKVSpec
    segments, Hq, Hkv, D, page, least, window, keep, chunk, with_sink, biased = step
    names = ("tc_attention_min_rows", "tc_pairs_min_units", "tc_pairs_units_a_tile", "tc_pairs_min_tiles", "tc_unit_min_tiles")
    saved = [getattr(kernels, name) for name in names]
    request.addfinalizer(lambda: [setattr(kernels, name, value) for name, value in zip(names, saved)])
    for name, value in zip(names, (2, 0 if pairs else None, {64: 0, 128: 0}, least, least)):
        setattr(kernels, name, value)
    batch, kv = paged_scenario(segments, num_kv_heads=Hkv, head_dim=D, page_size=page, dtype=torch.bfloat16, device="cpu", seed=31,
                               window=window, tc_min_key_tiles=least)
    kv = dataclasses.replace(kv, spec=PagedKVSpec(Hkv, D, window, None, keep, chunk) if chunk or keep else kv.spec)
    g = torch.Generator().manual_seed(32)
    q = torch.randn(batch.num_tokens, Hq * D, generator=g).to(torch.bfloat16)
    sink = 3.0 * torch.randn(Hq, generator=g) if with_sink else None
    slopes, cap = (0.02 * torch.rand(Hq, generator=g), 20.0) if biased else (None, None)
    ref = torch.zeros(batch.num_tokens, Hq * D, dtype=torch.bfloat16)
    REF.paged_attention(q, batch, kv, ref, Hq, D ** -0.5, sink=sink, score_cap=cap, slopes=slopes)
    if window and not keep:                                   # a windowed cache entry has given up what lies behind
        for i, (cached, _) in enumerate(segments):
            kv.block_table[i, :max(0, cached - window + 1) // page] = -1
    place = lambda t: None if t is None else t.to(DEV)
    ws = Workspace(DEV)
    first = None
    for _ in range(2):                                        # the tickets of the first call must be zero again
        out = torch.full((batch.num_tokens, Hq * D), float("nan"), dtype=torch.bfloat16, device=DEV)
        kernels.paged_attention(q.to(DEV), batch_to(batch, DEV), clone_kv(kv, DEV), out, Hq, D ** -0.5, ws, sink=place(sink), score_cap=cap,
                                slopes=place(slopes))
        kernels.check_errors()
        assert ("attn.pairs_tickets" in ws._buffers) == pairs
        assert_close(out, ref, TOL)
        assert first is None or torch.equal(first, out)       # the same bits, whichever block finishes first
        first = out
    tickets = ws._buffers["attn.pairs_tickets" if pairs else "attn.tc_tickets"]
    assert int(tickets.abs().sum()) == 0


def test_a_row_whose_maximum_grows_with_every_tile(kernels, request):
    """Keys that match a query better and better: O is multiplied by 2^(m_old - m_new) after every tile, from scores that differ by
    far more than a float's exponent, and the last key alone remains."""
    from kvcache_b200.engine.workspace import Workspace
    names = ("tc_attention_min_rows", "tc_pairs_min_units", "tc_pairs_units_a_tile")
    saved = [getattr(kernels, name) for name in names]
    request.addfinalizer(lambda: [setattr(kernels, name, value) for name, value in zip(names, saved)])
    kernels.tc_attention_min_rows, kernels.tc_pairs_min_units, kernels.tc_pairs_units_a_tile = 2, 0, {64: 0, 128: 0}
    for D in (64, 128):
        batch, kv = paged_scenario([(1000, 300)], num_kv_heads=1, head_dim=D, page_size=16, dtype=torch.bfloat16, device="cpu", seed=7)
        q = torch.ones(300, 2 * D, dtype=torch.bfloat16)
        for pos in range(1300):
            kv.k_pages[int(kv.block_table[0, pos // 16]), 0, pos % 16] = 0.02 * (pos - 650)
        ref, out = torch.zeros(300, 2 * D, dtype=torch.bfloat16), torch.zeros(300, 2 * D, dtype=torch.bfloat16, device=DEV)
        REF.paged_attention(q, batch, kv, ref, 2, 1.0)
        kernels.paged_attention(q.to(DEV), batch_to(batch, DEV), clone_kv(kv, DEV), out, 2, 1.0, Workspace(DEV))
        kernels.check_errors()
        assert_close(out, ref, TOL)


# (heads of, heads, segments, window, kernel): both sides of every line of the rule
ROUTES = [(64, 14, [(0, 400)], None, "attention_units"), (64, 14, [(2048, 1024)], None, "attention_pairs"), (64, 4, [(2048, 2048)], None, "attention_units"),
          (64, 14, [(0, 2048)], None, "attention_units"), (64, 28, [(2048, 2048)], 256, "attention_units"), (64, 28, [(2048, 2048)], 1024, "attention_pairs"),
          (64, 14, [(2048, 130)], None, "attention_units"), (64, 2, [(8000, 200)], None, None), (64, 2, [(2048, 200)], 256, "attention_units"),
          (128, 16, [(0, 800)], None, "attention_units"), (128, 16, [(2048, 512)], None, "attention_pairs"), (128, 2, [(2048, 512)], None, "attention_units"),
          (128, 16, [(0, 512)] * 4, None, "attention_units"), (128, 32, [(0, 512)] * 4, None, "attention_pairs"), (128, 8, [(2048, 2048)], 256, "attention_units"),
          (128, 2, [(2048, 130)], None, "attention_units")]


@pytest.mark.parametrize("route", ROUTES)
def test_which_kernel_a_portion_takes(kernels, route):
    from kvcache_b200.engine.workspace import Workspace
    D, H, segments, window, form = route
    batch, kv = paged_scenario(segments, num_kv_heads=2, head_dim=D, page_size=16, dtype=torch.bfloat16, device=DEV, seed=3, window=window)
    q = torch.randn(batch.num_tokens, H * D, device=DEV).to(torch.bfloat16)
    before, names = dict(kernels.launch_forms), kernels.launch_counts["attention_tc"]
    kernels.paged_attention(q, batch, kv, torch.empty_like(q), H, D ** -0.5, Workspace(DEV))
    kernels.check_errors()
    assert {f for f, n in kernels.launch_forms.items() if n > before.get(f, 0)} == ({form} if form else set())
    assert kernels.launch_counts["attention_tc"] == names + (form is not None)

"""Latent attention of portions with keys and values expanded first: the lists of its planner (no GPU), and the way from
queries to gated heads (gather and rotation, expansion, csrc/attention_pairs.cu) against float64."""
import math

import numpy as np
import pytest
import torch

from helpers import assert_close, batch_to, clone_kv, paged_scenario

DEV = "cuda:0"
TOL = 1e-2                 # q, keys, values, probabilities and results are rounded to 8 bits of mantissa: 2^-9 each


@pytest.mark.parametrize("window", [0, 1, 129, 300])
@pytest.mark.parametrize("segments", [[(0, 64)], [(0, 128), (127, 300)], [(1000, 200), (0, 257), (128, 64)], [(5, 2048)], [(3000, 65)]])
def test_lists_cover_every_key_that_a_row_sees(segments, window):
    from kvcache_b200.kernels.latent_plan import EXPAND_MIN_ROWS, LatentExpandPlanner
    planner = LatentExpandPlanner(window)
    arrays, counts = planner.plan(np.asarray([s for s, _ in segments]), np.asarray([n for _, n in segments]))
    room = planner.sections(sum(n for _, n in segments), len(segments))
    assert all(len(a) <= room[name] for name, a in arrays.items())
    blocks, key_row, pairs = arrays["blocks"].reshape(-1, 2), arrays["key_row"], arrays["pairs"].reshape(-1, 2)
    assert counts == {"blocks": len(blocks), "pairs": len(pairs)} and len(blocks) > 0
    for i, (start, count) in enumerate(segments):
        for key in range(max(0, start - window + 1) if window else 0, start + count):
            row = key_row[i] + key
            assert tuple(blocks[row // 128]) == (i, key // 128 * 128)        # a block starts at a multiple of 128 keys
        assert sorted(r for s, r in pairs if s == i) == list(range(0, count, 256))
    few = [(s, n) for s, n in segments] + [(10, EXPAND_MIN_ROWS - 1)]
    assert planner.plan(np.asarray([s for s, _ in few]), np.asarray([n for _, n in few]))[1] == {"blocks": 0, "pairs": 0}
    assert planner.plan(np.asarray([40000]), np.asarray([100]))[1]["blocks"] == (0 if not window else 2 + (window > 1) + (window > 200))


def test_weights_of_the_expansion_are_held_where_a_kernel_set_takes_the_sizes():
    from kvcache_b200.kernels.latent_plan import LatentAttentionPlanner, LatentExpandPlanner
    from kvcache_b200.parts.latent_attention import LatentAttention
    from kvcache_b200.parts.position import RotaryHalf

    class Kernels:
        def latent_attention_planner(self, *sizes): return LatentAttentionPlanner(sizes[0], 148)
        def latent_expand_planner(self, dim, vdim, rot_dim, kv_rank, window=None): return LatentExpandPlanner(0) if dim == 64 else None

    for dim, dtype in ((64, "bfloat16"), (48, "bfloat16"), (64, "float32")):
        part = LatentAttention(96, 3, dim, 16, dim, 40, 24, scale=0.1, eps=1e-6, position=RotaryHalf(16, 10000.0, 64), prefix="l.", dtype=dtype)
        g = torch.Generator().manual_seed(1)
        tensors = {name: torch.randn(*spec.shape, generator=g).to(getattr(torch, dtype)) for name, spec in part.tensor_specs().items()}
        for _ in range(2):                                     # also after weights have been bound anew
            part.bind(tensors, torch.device("cpu"))
            read, uv = part.weight_bytes(), part.w_uv.clone()
            assert part.w_ukv is None
            expands = dim == 64 and dtype == "bfloat16"
            for _ in range(2):
                assert len(part.step_planners(Kernels())) == 1 + expands
            assert (part.w_ukv is not None) == expands and part.weight_bytes() == read and torch.equal(part.w_uv, uv)
            if expands:
                assert torch.equal(part.w_ukv, torch.cat([tensors["l.uk"], tensors["l.uv"]])) and part.w_uv.data_ptr() == part.w_ukv[3 * dim:].data_ptr()


CASES = [
    # (segments, heads, dim, rot, rank, page, extra columns of q's rows, window, sink, one gate a head)
    ([(0, 64)], 3, 64, 16, 64, 16, 0, None, False, False),
    ([(0, 129), (200, 64)], 2, 128, 64, 96, 8, 0, None, True, False),
    ([(1000, 300), (37, 255), (0, 128)], 5, 64, 32, 256, 16, 40, None, False, True),
    ([(130, 700)], 4, 128, 48, 64, 64, 24, None, False, False),
    ([(900, 500), (5, 90)], 2, 64, 64, 72, 16, 0, 200, True, False),
    ([(300, 257)], 3, 128, 32, 128, 16, 8, 1, False, True),
    # the first key that is seen lies within a block of 128, and the pages before it have been given back
    ([(1000, 300), (900, 64)], 2, 64, 32, 64, 16, 0, 200, False, False),
    ([(2048, 100), (77, 130)], 3, 128, 16, 64, 8, 0, 1000, True, False),
    ([(0, 2000)], 14, 64, 32, 256, 16, 0, None, False, False),        # many pieces: streams divided and added up
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES)
def test_expanded_latent_attention(case):
    from kvcache_b200.engine.workspace import Workspace
    from kvcache_b200.kernels.api import CudaKernels
    from kvcache_b200.parts.base import StepPlan
    segments, H, dim, R, C, page, extra, window, with_sink, per_head = case
    kernels = CudaKernels(DEV)
    g = torch.Generator().manual_seed(3)
    rand = lambda *shape: torch.randn(*shape, generator=g)
    batch, kv = paged_scenario(segments, num_kv_heads=1, head_dim=C + R, page_size=page, dtype=torch.bfloat16, device="cpu", seed=4, window=window)
    T = batch.num_tokens
    half = max(1, R // 2 - (8 if R > 16 else 0))                       # not all of the rotated part turns
    angle = torch.outer(torch.arange(4096.0), 10000.0 ** (-torch.arange(half) / half))
    cos, sin = torch.cos(angle).contiguous(), torch.sin(angle).contiguous()
    q = rand(T, H * (dim + R) + extra).to(torch.bfloat16)
    w = (rand(2 * H * dim, C) * C ** -0.5).to(torch.bfloat16)
    gate = rand(T, (H if per_head else H * dim) + 16).to(torch.bfloat16)
    sink = rand(H) if with_sink else None
    scale = (dim + R) ** -0.5

    want = torch.empty(T, H, dim, dtype=torch.float64)
    qd = q[:, :H * (dim + R)].double().view(T, H, dim + R)
    c, s = cos[batch.positions.long()].double()[:, None], sin[batch.positions.long()].double()[:, None]
    lo, hi = qd[..., dim:dim + half], qd[..., dim + half:dim + 2 * half]
    qd = torch.cat([qd[..., :dim], lo * c - hi * s, hi * c + lo * s, qd[..., dim + 2 * half:]], dim=-1)
    at = 0
    held = torch.zeros(kv.k_pages.shape[:-1], dtype=torch.bool)
    for i, (start, n) in enumerate(segments):
        L = start + n
        pages = kv.block_table[i, :-(-L // page)].long()
        rows = kv.k_pages[pages, 0].reshape(-1, C + R)[:L].double()
        at_key = torch.arange(len(pages) * page)
        held[pages, 0] |= ((at_key < L) & (at_key >= (max(0, start - window + 1) if window else 0))).view(-1, page)
        keys = torch.cat([(rows[:, :C] @ w[:H * dim].double().t()).view(L, H, dim), rows[:, None, C:].expand(L, H, R)], dim=-1)
        values = (rows[:, :C] @ w[H * dim:].double().t()).view(L, H, dim)
        pos, j = start + torch.arange(n)[:, None], torch.arange(L)[None]
        seen = (j <= pos) & (pos - j < (window or L))
        for h in range(H):
            score = (qd[at:at + n, h] @ keys[:, h].t() * scale).masked_fill(~seen, -math.inf)
            if sink is not None:
                score = torch.cat([score, sink[h].double().expand(n, 1)], dim=1)
            want[at:at + n, h] = torch.softmax(score, dim=1)[:, :L] @ values[:, h]
        at += n
    sig = torch.sigmoid(gate[:, 8:8 + (H if per_head else H * dim)].double())
    want = (want * (sig[:, :, None] if per_head else sig.view(T, H, dim))).reshape(T, H * dim)

    kv.k_pages[~held] = float("nan")                                   # rows that no request holds, or sees any more, must not be used
    if window:
        for i, (start, _) in enumerate(segments):
            kv.block_table[i, :max(0, start - window + 1) // page] = -1        # as the cache gives pages back
    planner = kernels.latent_expand_planner(dim, dim, R, C, window)
    arrays, counts = planner.plan(np.asarray([a for a, _ in segments]), np.asarray([n for _, n in segments]))
    place = lambda t: None if t is None else t.to(DEV)
    batch = batch_to(batch, DEV)
    batch.plans[planner.name] = StepPlan({k: torch.from_numpy(a.copy()).to(DEV) for k, a in arrays.items()}, counts)
    ws, bits = Workspace(DEV), None
    for _ in range(2):
        out = torch.full((T, H * dim), float("nan"), dtype=torch.bfloat16, device=DEV)
        assert kernels.latent_expanded_attention(q.to(DEV), w.to(DEV), batch, clone_kv(kv, DEV), out, H, dim, scale, ws, cos.to(DEV), sin.to(DEV),
                                                 (gate.to(DEV), 8), per_head, window, place(sink))
        kernels.check_errors()
        assert_close(out, want, TOL)
        assert bits is None or torch.equal(bits, out)
        bits = out
    assert int(ws._buffers["attn.pairs_tickets"].abs().sum()) == 0

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


@pytest.mark.parametrize("dtype,out_dtype,N,K", [
    (torch.float32, torch.float32, 1153, 132), (torch.float32, torch.float32, 896, 4864), (torch.float32, torch.float32, 9728, 100),
    (torch.float32, torch.float32, 40, 77), (torch.float32, torch.float32, 1153, 333), (torch.float32, torch.float32, 9728, 77),
    (torch.bfloat16, torch.bfloat16, 1153, 136), (torch.bfloat16, torch.float32, 9728, 104), (torch.bfloat16, torch.bfloat16, 9728, 100),
    (torch.bfloat16, torch.float32, 1153, 333)])
def test_float32_product_rows_do_not_depend_on_the_tile(kernels, dtype, out_dtype, N, K):
    """Every number of rows at the edges of the tiles and of the rule that picks one (1,153 and 9,728 outputs meet all five), K that
    comes in 16 bytes at a time and K that does not: close to 64 bits, and each row bit for bit what it is in the largest step (one
    chain over k, whatever the tile)."""
    from kvcache_b200.kernels.api import _dtype_code, _ptr
    g = torch.Generator().manual_seed(31)
    x, w, bias = torch.randn(1001, K, generator=g).to(dtype), torch.randn(N, K, generator=g).to(dtype), torch.randn(N, generator=g)
    xd, wd, bd = x.to(DEV), w.to(DEV), bias.to(DEV)

    def product(M):
        out = torch.full((M, N), float("nan"), dtype=out_dtype, device=DEV)
        with kernels.on_current_stream():
            assert kernels._gemm_simt.kvb_gemm_simt(_dtype_code(dtype), _dtype_code(out_dtype), _ptr(xd), _ptr(wd), _ptr(bd), _ptr(out), M, N, K,
                                                    kernels._stream()) == 0
        return out

    full, want = product(1001), x.double() @ w.double().t() + bias.double()
    # A chain of K rounded multiply-adds: at most K 2^-24 times the sum of magnitudes, which for normal numbers is 0.64 K; then a rounding
    # to 8 significant bits in bfloat16, at most half of the last of them: 2^-8 of the result.
    bound = K * 2.0 ** -24 * ((x.abs().double() @ w.abs().double().t()).max().item() + 5.0)
    bound += want.abs().max().item() * 2.0 ** -8 if out_dtype == torch.bfloat16 else 0.0
    assert (full.double().cpu() - want).abs().max().item() <= bound
    for M in (1, 4, 5, 16, 17, 48, 49, 64, 65, 129, 513):
        assert torch.equal(product(M), full[:M]), M


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_products_with_a_matrix_made_by_the_launch_before(dtype):
    """W may be the result of the launch before: nothing of it is read while that one still runs."""
    from kvcache_b200.kernels.api import CudaKernels
    kernels = CudaKernels(DEV, bf16_gemm="simt")             # a launch that lets the next one start before it has ended
    g = torch.Generator(device=DEV).manual_seed(33)
    H, N, K = 8, 512, 128
    rand = lambda *s: torch.randn(*s, generator=g, device=DEV).to(dtype)
    x, w = rand(40, K), torch.zeros(H * N, K, dtype=dtype, device=DEV)
    heads_x, heads_out = rand(40, H * K), torch.empty(40, H * N, dtype=dtype, device=DEV)
    out = torch.empty(40, H * N, dtype=dtype, device=DEV)
    for _ in range(8):
        a, b = rand(H * N, 320), rand(K, 320)
        kernels.linear(a, b, w)
        kernels.linear(x, w, out)
        kernels.linear(a, b, w)
        kernels.head_linear(heads_x, w.view(H, N, K), heads_out)
        torch.cuda.synchronize()
        after, heads_after = torch.empty_like(out), torch.empty_like(heads_out)
        kernels.linear(x, w, after)
        torch.cuda.synchronize()
        kernels.head_linear(heads_x, w.view(H, N, K), heads_after)
        torch.cuda.synchronize()
        assert torch.equal(out, after) and torch.equal(heads_out, heads_after)
        w.zero_()
        torch.cuda.synchronize()


ROWS32 = [
    ([(0, 1), (63, 1), (64, 1), (500, 1)], 14, 2, 64, 64, 16, {}),                       # decoded tokens at the edge of a key tile
    ([(0, 65), (64, 64), (127, 3), (5, 1)], 6, 2, 64, 64, 16, {}),                       # tiles of rows that end inside a segment
    ([(700, 1), (3, 90), (0, 33)], 6, 2, 48, 80, 8, dict(window=100, keep_first=5)),     # kept keys beside a window; unequal sizes
    ([(700, 70), (3, 90)], 3, 1, 20, 4, 16, dict(chunk=48)),
    ([(0, 130), (900, 300)], 16, 2, 128, 128, 32, dict(window=64)),
    ([(200, 700)], 2, 2, 128, 100, 64, {}),
    ([(30, 1), (3, 2)], 2, 1, 16, 16, 16, {}),                                           # shared memory right below what needs no asking for
    ([(7 * i % 130, 1 + i % 2) for i in range(90)], 8, 4, 64, 64, 16, {}),               # many segments of few rows: eight a block ...
    ([(7 * i % 130, 1 + i % 3) for i in range(50)], 20, 4, 68, 128, 16, dict(window=40, keep_first=3)),      # ... and one stage of keys
]


@pytest.mark.parametrize("scenario", ROWS32)
@pytest.mark.parametrize("options", [False, True])
def test_float32_attention_tiles(kernels, scenario, options, monkeypatch):
    monkeypatch.setattr(kernels, "ROWS32_MIN", 4)                                        # narrower heads than the dispatch gives it
    monkeypatch.setattr(kernels, "ROWS32_MIN_SHARED", 4)
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


def _scan_exact(mode, lens, q, k, v, a, b, u, c, state, scale, dtype=torch.float64):
    """The recurrence token by token in 64 bits; q, k [T, G, D], v [T, H, Dv], a (and u, c) [T, H, D], b [T, H]."""
    H, G = v.shape[1], q.shape[1]
    outs, ends, at = [], [], 0
    q, k, v, a, b, u, c = (x.to(dtype) for x in (q, k, v, a, b, u, c))
    for i, n in enumerate(lens):
        S = state[i].to(dtype)
        for t in range(at, at + n):
            qt, kt = q[t].repeat_interleave(H // G, 0), k[t].repeat_interleave(H // G, 0)
            if mode == "gated_delta":
                S = a[t][:, :, None] * S
                S = S + kt[:, :, None] * (b[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, kt)))[:, None]
            elif mode == "delta_rule":
                S = a[t][:, :, None] * S - c[t][:, :, None] * torch.einsum("hdv,hd->hv", S, u[t])[:, None] \
                    + kt[:, :, None] * v[t][:, None]
            elif mode == "channel_decay":
                S = a[t][:, :, None] * S + kt[:, :, None] * v[t][:, None]
            else:
                S = a[t][:, :1, None] * S + b[t][:, None, None] * kt[:, :, None] * v[t][:, None]
            outs.append(torch.einsum("hdv,hd->hv", S, qt) * scale)
        ends.append(S)
        at += n
    return torch.stack(outs), torch.stack(ends)


MODES = ["gated_delta", "delta_rule", "channel_decay", "head_decay"]


def _scan_inputs(mode, lens, H, G, D, Dv, decay):
    """q, k, v, a, b, u, c, states of the segments and two more slots; `decay(random numbers)`: the decays."""
    g = torch.Generator().manual_seed(51)
    T = sum(lens)
    rand = lambda *s: torch.randn(*s, generator=g)
    if mode == "delta_rule":
        G = H
    q, k, v, b = rand(T, G, D), rand(T, G, D), rand(T, H, Dv), torch.sigmoid(rand(T, H))
    k = k / k.norm(dim=-1, keepdim=True)
    a = decay(torch.rand(T, H, D, generator=g))
    if mode == "head_decay":
        a = a[:, :, :1].expand(T, H, D).contiguous()
    u = rand(T, H, D)
    u = u / u.norm(dim=-1, keepdim=True)
    c = u * torch.rand(T, H, D, generator=g)
    return q, k, v, a, b, u, c, rand(len(lens) + 2, H, D, Dv)


def _scan_chunks(kernels, mode, lens, q, k, v, a, b, u, c, state, slots):
    """What the scan over chunks makes of them: read-outs [T, H, Dv] (times 0.5) and all slots' states."""
    from kvcache_b200.engine.workspace import Workspace
    from kvcache_b200.parts.base import StepBatch
    (T, H, Dv), (G, D) = v.shape, q.shape[1:]
    if mode == "head_decay":
        rows, gates, cols = torch.cat([v.flatten(1), k.flatten(1), q.flatten(1)], 1), torch.cat([a[:, :, 0], b], 1), (H * Dv + G * D, H * Dv, 0)
    else:
        rows, cols = torch.cat([q.flatten(1), k.flatten(1), v.flatten(1)], 1), (0, G * D, 2 * G * D)
        gates = torch.cat([a.flatten(1)] + ([b] if mode == "gated_delta" else [u.flatten(1), c.flatten(1)] if mode == "delta_rule" else []), 1)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    batch = StepBatch(T, len(lens), 0, None, None, None, i32([sum(lens[:i]) for i in range(len(lens))]), i32(lens), None, i32(slots), None,
                      max_q_len=max(lens))
    memory, out = state.clone().to(DEV), torch.full((T, H * Dv), float("nan"), device=DEV)
    kernels._chunk_scan(mode, rows.contiguous().to(DEV), cols, G, gates.contiguous().to(DEV), 0.5, batch, memory, out, H, D, Dv, Workspace(DEV))
    kernels.check_errors()
    return out.view(-1, H, Dv).cpu(), memory.cpu()


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("lens,H,G,D,Dv", [([16, 1, 17, 15], 2, 1, 64, 16), ([64], 3, 3, 65, 24), ([33, 100], 4, 2, 128, 40), ([300], 1, 1, 16, 7),
                                           ([2, 31], 3, 3, 37, 130)])
def test_scan_in_chunks(kernels, mode, lens, H, G, D, Dv):
    """Every form of the scan over chunks of sixteen tokens: remainders of chunks, channels and values, shared queries and keys,
    decays of zero and near it, states that are not empty; and a segment alone gives the bits it gives beside others."""
    T, S = sum(lens), len(lens)
    *tokens, state = _scan_inputs(mode, lens, H, G, D, Dv, lambda r: torch.exp(-0.6 * r ** 3))
    tokens[3][T // 2], tokens[3][T // 3] = 0.0, 1e-30
    slots = list(range(S, 0, -1))
    out, memory = _scan_chunks(kernels, mode, lens, *tokens, state, slots)
    want, ends = _scan_exact(mode, lens, *tokens, state[slots], 0.5)
    untouched = [i for i in range(S + 2) if i not in slots]
    assert torch.equal(memory[untouched], state[untouched])
    # Rounded sums of about 4 D + 64 products, of independent sign, make a result or state: sqrt(4 D + 64) 2^-24 is 1.4e-6 at D = 128.
    for got, ref in ((out, want), (memory[slots], ends)):
        assert ((got.double() - ref).norm() / ref.norm()).item() <= 1.4e-6
    alone, memory_alone = _scan_chunks(kernels, mode, lens[:1], *(t[:lens[0]] for t in tokens), state, slots[:1])
    assert torch.equal(alone, out[:lens[0]]) and torch.equal(memory_alone[slots[0]], memory[slots[0]])


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("rate", [0.05, 0.6, 3.0])
@pytest.mark.parametrize("lens,D", [([200, 37], 64), ([116, 52], 128)])
def test_scan_in_chunks_rounds_no_worse_than_a_walk_over_tokens(kernels, mode, rate, lens, D):
    """Slow, mixed and fast decays: the distance from 64 bits is at most that of the recurrence taken token by token in float32, with a
    tenth for the luck of roundings (some ten thousand numbers share it)."""
    *tokens, state = _scan_inputs(mode, lens, 3, 3, D, 32, lambda r: torch.exp(-rate * r))
    slots = [0, 1]
    exact, walk = (_scan_exact(mode, lens, *tokens, state[slots], 0.5, dtype) for dtype in (torch.float64, torch.float32))
    out, memory = _scan_chunks(kernels, mode, lens, *tokens, state, slots)
    for got, over_tokens, ref in zip((out, memory[slots]), walk, exact):
        off = lambda x: ((x.double() - ref).norm() / ref.norm()).item()
        assert off(got) <= 1.1 * off(over_tokens)


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("D", [64, 128])
def test_scan_in_chunks_within_bounded_scratch(kernels, mode, D, monkeypatch):
    """Scratch for one chunk, for two and for three at a time: the same bits as for all of them, through segments that end inside a run,
    with one and that take several; and no more of it than the bound."""
    lens, H, Dv = [40, 1, 16, 100, 33], 2, 24
    *tokens, state = _scan_inputs(mode, lens, H, H, D, Dv, lambda r: torch.exp(-0.5 * r))
    slots = [4, 2, 0, 1, 6]
    out, memory = _scan_chunks(kernels, mode, lens, *tokens, state, slots)
    code, lib = kernels.CHUNK_MODES[mode], kernels._scan_chunk
    size = 4 * H * (lib.kvb_chunk_record_floats(code, D) + lib.kvb_chunk_shared_floats(code, D))
    for held in (1, 2, 3):
        monkeypatch.setattr(kernels, "CHUNK_SCRATCH_BYTES", held * size)
        before = kernels.launches
        got = _scan_chunks(kernels, mode, lens, *tokens, state, slots)
        assert torch.equal(got[0], out) and torch.equal(got[1], memory)
        assert kernels.launches - before == -(-(sum(lens) // 16 + len(lens)) // held) * (3 if mode == "delta_rule" else 2) - 1


INPUTS = {"gated_delta": "qkvab", "delta_rule": "qkvauc", "channel_decay": "qkva", "head_decay": "qkvab"}


@pytest.mark.parametrize("mode,what", [(mode, what) for mode in MODES for what in INPUTS[mode]])
def test_scan_in_chunks_keeps_a_token_from_those_before_it(kernels, mode, what):
    """An infinite or undefined number in any of a token's inputs: the tokens before it give the bits they give without it, and such a
    value leaves the other value channels' alone."""
    lens, H, D, Dv, at, i = [40], 2, 64, 24, 29, "qkvabuc".index(what)
    *tokens, state = _scan_inputs(mode, lens, H, H, D, Dv, lambda r: torch.exp(-r))
    out, memory = _scan_chunks(kernels, mode, lens, *tokens, state, [1])
    sound = tokens[i]
    for number in (float("inf"), float("nan")):
        tokens[i] = sound.clone()
        if mode == "head_decay" and what == "a":
            tokens[i][at] = number                                       # one decay for all channels of a head
        else:
            tokens[i][at].view(-1)[0 if what == "b" else 5] = number
        bad, bad_memory = _scan_chunks(kernels, mode, lens, *tokens, state, [1])
        assert torch.equal(bad[:at], out[:at])
        assert not torch.isfinite(bad[at:]).all()
        if what == "v":
            others = [c for c in range(Dv) if c != 5]
            assert torch.equal(bad[..., others], out[..., others]) and torch.equal(bad_memory[..., others], memory[..., others])


@pytest.mark.parametrize("M", [17, 32, 33, 65, 300])
@pytest.mark.parametrize("H,N,K,rot,gate", [(3, 512, 128, 64, None), (3, 128, 512, 0, "channel"), (5, 136, 72, 24, "head"), (20, 8, 8, 3, None)])
def test_head_products_in_tiles(kernels, M, H, N, K, rot, gate):
    """More than 16 rows: remainders of rows, outputs and K, rotated columns (an odd number of them not rotated), both kinds of gate;
    and every row bit for bit what sixteen rows at a time give."""
    g = torch.Generator().manual_seed(61)
    rot_half = rot // 4
    rot_pad = rot + -rot % 8 if rot else 0                                   # rows of x and of the result start on 16 bytes
    if rot_pad != rot:
        rot = rot_pad
    x = torch.randn(M, H * (K + rot), generator=g).to(torch.bfloat16)
    w = torch.randn(H, N, K, generator=g).to(torch.bfloat16)
    gates = torch.randn(M, 8 + H * (N + rot), generator=g).to(torch.bfloat16)
    positions = torch.randperm(400, generator=g)[:M].to(torch.int32)
    cos, sin = torch.randn(400, max(rot_half, 1), generator=g), torch.randn(400, max(rot_half, 1), generator=g)

    def run(rows):
        out = torch.full((rows.stop - rows.start, H * (N + rot)), float("nan"), dtype=torch.bfloat16, device=DEV)
        more = {}
        if rot:
            more["rotate"] = (cos.to(DEV), sin.to(DEV), positions[rows].contiguous().to(DEV))
        if gate:
            more.update(gate=(gates[rows].contiguous().to(DEV), 8), gate_per_head=gate == "head")
        kernels.head_linear(x[rows].contiguous().to(DEV), w.to(DEV), out, **more)
        kernels.check_errors()
        return out.cpu()

    out = run(slice(0, M))
    assert torch.equal(out, torch.cat([run(slice(i, min(i + 16, M))) for i in range(0, M, 16)]))
    xs = x.view(M, H, K + rot).double()
    want = torch.einsum("mhk,hnk->mhn", xs[:, :, :K], w.double())
    if gate:
        logits = gates[:, 8:8 + H].double()[:, :, None] if gate == "head" else gates[:, 8:].double().view(M, H, N + rot)[:, :, :N]
        want = want * torch.sigmoid(logits)
    # float32 sums of K products, rounded to 8 bits of fraction once.
    assert_close(out.view(M, H, N + rot)[:, :, :N], want, 2.0 ** -8 + K * 2.0 ** -22)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,H,Dv,parts", [(3, 5, 4, 1), (7, 3, 64, 3), (130, 2, 128, 2), (5, 64, 64, 1)])
def test_gated_norms_in_fours(kernels, dtype, T, H, Dv, parts):
    """Rows that start on 16 bytes go four numbers at a time; the same rows one column further go one at a time: the same results but
    for the order of a sum of W squares (at most W 2^-24 of it) and one rounding to the result's type."""
    W = H * Dv
    rand = lambda *s: torch.randn(*s, generator=torch.Generator(device=DEV).manual_seed(len(s) * 7 + s[0]), device=DEV)
    o, x, skip, w, head_w = rand(T, W), rand(T, W + 8), rand(H), rand(W), rand(Dv)
    aligned, shifted = torch.zeros(T, W + 8, device=DEV), torch.zeros(T, W + 9, device=DEV)
    aligned[:, 4:4 + W] = rand(T, W) * 3
    shifted[:, 5:5 + W] = aligned[:, 4:4 + W]
    results = []
    for gate, col, width in ((aligned, 4, W + 12), (shifted, 5, W + 13)):
        part, head = (torch.full((T, width), 7.0, dtype=dtype, device=DEV) for _ in range(2))
        kernels.gate_part_norm(o, x, skip, (gate, col), w, 1e-6, 0.5, part, col + 4, H, Dv, parts)
        kernels.head_norm_gate(o, head_w, 1e-6, (gate, col), "silu", 0.5, head, col + 4, H, Dv)
        for r in (part, head):
            assert (r[:, :col + 4] == 7.0).all() and (r[:, col + 4 + W:] == 7.0).all()
        results.append((part[:, col + 4:col + 4 + W], head[:, col + 4:col + 4 + W]))
    for a, b in zip(*results):
        assert_close(a, b, 2.0 ** -7 if dtype == torch.bfloat16 else 1e-6 + W * 2.0 ** -24)

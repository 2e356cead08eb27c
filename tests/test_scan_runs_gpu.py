"""Scans whose decays alone carry the state, walked in several runs of chunks at once (csrc/scan_chunk.cu), against a walk over tokens in
64 bits and against one run."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def kernels():
    from kvcache_b200.kernels.api import CudaKernels
    return CudaKernels(DEV)


def _int32(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


def _scan(kernels, mode, rows, gates, G, counts, memory, H, D, Dv, run_chunks):
    from kvcache_b200.engine.workspace import Workspace
    starts = [sum(counts[:i]) for i in range(len(counts))]
    batch = SimpleNamespace(seg_q_start=_int32(starts), seg_q_len=_int32(counts), seg_slot=_int32(list(range(len(counts)))), num_segments=len(counts),
                            num_tokens=sum(counts), max_q_len=max(counts))
    kernels.CHUNK_RUN_MAX_BLOCKS = {mode: 1 << 30} if run_chunks else {}
    kernels.CHUNK_RUN_MIN, kernels.CHUNK_RUN_BLOCKS, kernels.CHUNK_RUN_MIN_CHUNKS = run_chunks, 1 << 30, 0
    state, out = memory.clone(), torch.full((sum(counts), H * Dv), float("nan"), device=DEV)
    before = kernels.launches
    kernels._chunk_scan(mode, rows, (0, G * D, 2 * G * D), G, gates, 0.5, batch, state, out, H, D, Dv, Workspace(DEV))
    kernels.check_errors()
    assert kernels.launches - before == (3 if run_chunks else 1)        # records, ends, starts and the walk, one counted by the caller
    return out, state


@pytest.fixture(autouse=True)
def _settings(kernels):
    yield
    for name in ("CHUNK_RUN_MAX_BLOCKS", "CHUNK_RUN_MIN", "CHUNK_RUN_BLOCKS", "CHUNK_RUN_MIN_CHUNKS"):
        kernels.__dict__.pop(name, None)


# Lengths around the ends of chunks of 16 and of runs; head sizes that are no multiple of anything; heads that share keys.
CASES = [("channel_decay", 2, 2, 64, 128, [15, 16, 17, 96, 97, 95]), ("channel_decay", 3, 3, 40, 24, [200, 1, 333]), ("channel_decay", 1, 1, 128, 17, [530]),
         ("head_decay", 4, 1, 128, 64, [47, 48, 49, 160]), ("head_decay", 6, 2, 100, 40, [1, 400, 129]), ("head_decay", 20, 1, 33, 16, [257])]


@pytest.mark.parametrize("run_chunks", [1, 3, 5])
@pytest.mark.parametrize("mode,H,G,D,Dv,counts", CASES)
def test_runs_of_chunks_walked_at_once(kernels, mode, H, G, D, Dv, counts, run_chunks):
    g = torch.Generator().manual_seed(5)
    T = sum(counts)
    rows = torch.randn(T, 2 * G * D + H * Dv, generator=g)
    decay = 0.8 + 0.2 * torch.rand(T, H * D if mode == "channel_decay" else H, generator=g)
    decay[torch.rand(decay.shape, generator=g) < 0.002] = 0.0           # a decay of zero forgets all before it
    gain = torch.rand(T, H, generator=g)
    gates = decay if mode == "channel_decay" else torch.cat([decay, gain], dim=1)
    memory = torch.randn(len(counts), H, D, Dv, generator=g)
    want, state, at = torch.empty(T, H, Dv, dtype=torch.float64), memory.double().clone(), 0
    for i, n in enumerate(counts):
        S = state[i]
        for t in range(at, at + n):
            row = rows[t].double()
            q, k = (row[j * G * D:(j + 1) * G * D].view(G, D).repeat_interleave(H // G, 0) for j in (0, 1))
            kv = k[:, :, None] * row[2 * G * D:].view(H, 1, Dv)
            a = decay[t].double().view(H, -1, 1)
            S = a * S + (kv if mode == "channel_decay" else gain[t].double().view(H, 1, 1) * kv)
            want[t] = 0.5 * torch.einsum("hdv,hd->hv", S, q)
        state[i], at = S, at + n
    out, end = _scan(kernels, mode, rows.to(DEV), gates.contiguous().to(DEV), G, counts, memory.to(DEV), H, D, Dv, run_chunks)
    # Sums of up to a few hundred float32 terms of size one: 2^-24 each, in any order.
    assert (out.cpu().double().view(T, H, Dv) - want).abs().max() <= 2e-5 * want.abs().max()
    assert (end.cpu().double() - state).abs().max() <= 2e-5 * state.abs().max()


@pytest.mark.parametrize("mode,H,D,Dv", [("channel_decay", 2, 64, 32), ("head_decay", 2, 64, 32)])
def test_an_infinite_or_undefined_number_goes_where_it_goes_in_one_run(kernels, mode, H, D, Dv):
    g = torch.Generator().manual_seed(6)
    T = 700
    for value in (float("inf"), float("nan")):
        for where in (3, 40, 300, 699):
            rows = torch.randn(T, 2 * H * D + H * Dv, generator=g).to(DEV)
            gates = (0.3 + 0.6 * torch.rand(T, H * D if mode == "channel_decay" else H, generator=g)).to(DEV)     # products that run out of exponents
            if mode == "head_decay":
                gates = torch.cat([gates, torch.rand(T, H, generator=g).to(DEV)], dim=1).contiguous()
            rows[where, 2 * H * D + 5] = value
            memory = torch.randn(1, H, D, Dv, generator=g).to(DEV)
            memory[0, 1, 7, 9] = value
            one = _scan(kernels, mode, rows, gates, H, [T], memory, H, D, Dv, 0)
            many = _scan(kernels, mode, rows, gates, H, [T], memory, H, D, Dv, 4)
            for a, b in zip(one, many):
                assert torch.equal(torch.isfinite(a), torch.isfinite(b)) and torch.equal(torch.isnan(a), torch.isnan(b))
                ok = torch.isfinite(a)
                assert (a[ok] - b[ok]).abs().max() <= 2e-5 * a[ok].abs().max()


@pytest.mark.parametrize("mode,H,G,D,Dv", [("channel_decay", 7, 7, 64, 128), ("channel_decay", 2, 2, 100, 40), ("head_decay", 28, 1, 128, 64), ("head_decay", 3, 3, 64, 64)])
def test_a_segment_is_the_same_bits_beside_any_others(kernels, mode, H, G, D, Dv):
    """With the rule as it is: segments that are cut into runs and ones that are not, alone and in steps with others of any length, also
    more of them than would be cut if their number counted."""
    from kvcache_b200.engine.workspace import Workspace
    g = torch.Generator().manual_seed(9)
    counts = [1000, 383, 1, 900, 640, 385, 1000]
    starts, T, ws = [sum(counts[:i]) for i in range(len(counts))], sum(counts), Workspace(DEV)
    rows = torch.randn(T, 2 * G * D + H * Dv, generator=g).to(DEV)
    decay = 0.8 + 0.2 * torch.rand(T, H * D if mode == "channel_decay" else H, generator=g)
    gates = (decay if mode == "channel_decay" else torch.cat([decay, torch.rand(T, H, generator=g)], dim=1)).contiguous().to(DEV)
    memory = torch.randn(len(counts), H, D, Dv, generator=g).to(DEV)

    def scan(which):
        part = torch.cat([torch.arange(starts[i], starts[i] + counts[i]) for i in which]).to(DEV)
        mine = [counts[i] for i in which]
        batch = SimpleNamespace(seg_q_start=_int32([sum(mine[:i]) for i in range(len(mine))]), seg_q_len=_int32(mine), seg_slot=_int32(list(range(len(mine)))),
                                num_segments=len(mine), num_tokens=sum(mine), max_q_len=max(mine))
        state, out, before = memory[list(which)].contiguous(), torch.full((sum(mine), H * Dv), float("nan"), device=DEV), kernels.launches
        kernels._chunk_scan(mode, rows[part].contiguous(), (0, G * D, 2 * G * D), G, gates[part].contiguous(), 0.5, batch, state, out, H, D, Dv, ws)
        kernels.check_errors()
        return dict(zip(which, zip(out.split(mine), state))), kernels.launches - before

    want, cut = {}, set()
    for i in range(len(counts)):
        one, launches = scan([i])
        want.update(one)
        cut.add(launches == 3)
    assert cut == {True, False}
    for which in ([0, 6], [0, 3, 4, 5, 6], list(range(len(counts))), [2, 1, 3]):
        for i, (out, state) in scan(which)[0].items():
            assert torch.equal(out, want[i][0]) and torch.equal(state, want[i][1]), (which, i)

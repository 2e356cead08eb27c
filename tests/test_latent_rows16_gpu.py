"""Attention over shared key rows for single tokens (tiles of 16 rows, csrc/latent_flash.cu) at the edges of its forms: key sizes on both
sides of what its instances hold, runs of keys that end anywhere in a tile of 64, several splits, a window that starts within a tile."""
import dataclasses

import numpy as np
import pytest
import torch

from helpers import assert_close, batch_to, clone_kv, paged_scenario
from torch_kernels import TorchKernels

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TOL = 1e-2                 # bfloat16 queries, keys, probabilities and results, as in the other tests of this kernel


@pytest.fixture(scope="module")
def kernels():
    from kvcache_b200.kernels.api import CudaKernels
    return CudaKernels(DEV)


STEPS = ([(63, 1), (64, 1), (0, 1), (191, 1), (700, 1)], [(2000, 1)])


def _compare(kernels, H, Dk, Dv, window, steps=STEPS):
    from kvcache_b200.engine.workspace import Workspace
    from kvcache_b200.parts.base import StepPlan
    for segments in steps:
        batch, kv = paged_scenario(segments, num_kv_heads=1, head_dim=Dk, page_size=16, dtype=torch.bfloat16, device="cpu", seed=8, window=window)
        planner = kernels.latent_attention_planner(H, Dk, Dv, window)
        arrays, counts = planner.plan(np.asarray([s for s, _ in segments]), np.asarray([n for _, n in segments]))
        assert counts["bm"] == 16
        batch = dataclasses.replace(batch, plans={planner.name: StepPlan({k: torch.tensor(np.array(v), dtype=torch.int32) for k, v in arrays.items()}, counts)})
        g = torch.Generator().manual_seed(9)
        q = torch.randn(len(segments), H * Dk, generator=g).to(torch.bfloat16)
        for sink in (None, torch.randn(H, generator=g)):
            ref, got = torch.zeros(len(segments), H * Dv, dtype=torch.bfloat16), torch.full((len(segments), H * Dv), 7.0, dtype=torch.bfloat16, device=DEV)
            TorchKernels(wide=True).latent_attention(q, batch, kv, ref, H, Dv, Dk ** -0.5, sink=sink)
            held = clone_kv(kv, DEV)
            if window:
                for i, (start, _) in enumerate(segments):
                    held.block_table[i, :max(0, start - window + 1) // 16] = -1
            kernels.latent_attention(q.to(DEV), batch_to(batch, DEV), held, got, H, Dv, Dk ** -0.5, Workspace(DEV), sink=None if sink is None else sink.to(DEV))
            kernels.check_errors()
            assert_close(got, ref, TOL)


@pytest.mark.parametrize("window", [None, 70])
@pytest.mark.parametrize("H,Dk,Dv", [(16, 8, 8), (2, 16, 4), (1, 160, 128), (5, 168, 64), (14, 320, 256), (16, 328, 300), (16, 576, 512), (3, 576, 60), (2, 584, 512)])
def test_single_tokens_over_shared_key_rows(kernels, H, Dk, Dv, window):
    _compare(kernels, H, Dk, Dv, window)


@pytest.mark.parametrize("H,Dk,Dv", [(14, 152, 132), (16, 160, 144), (3, 160, 160), (16, 264, 260), (5, 304, 272), (16, 320, 288), (2, 320, 320)])
def test_values_wider_than_an_instance_of_their_key_size(kernels, H, Dk, Dv):
    """More value columns than the instance that their key size leads to adds up: 128 for keys of up to 160 numbers, 256 up to 320.  Cut into
    several splits, and more requests than the plan wants blocks, a single one."""
    _compare(kernels, H, Dk, Dv, None, (*STEPS, [(17 * i % 90, 1) for i in range(2 * 148 + 4)]))

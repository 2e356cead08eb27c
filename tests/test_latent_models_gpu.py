"""Latent layers whose heads are of sizes that portions expand (64 and 128), through the engine in bfloat16: windows that are no multiple of a
block of expanded keys, a layer that reads another one's latent through a narrower window, portions that start anywhere, graphs."""
import os

import pytest
import torch

import plain_kakipel
import plain_karorax
import replay_modes
from helpers import assert_close, make_runner, random_tokens
from kakipel_configs import DENSE, _layer as kaki_layer, _mixer
from karorax_configs import _dense, _latent, _layer, make_karorax_folder
from test_karorax_gpu import _spread, assert_model_close

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
KARORAX = {
    "architecture": "Karorax", "vocab": 211, "width": 128, "norm": {"eps": 1e-6}, "logit_softcap": 20.0,
    "layers": [
        _layer(_latent(3, 64, 16, 64, 64, 0.11, 100, (50000.0, 16)), _dense(192)),
        _layer(_latent(2, 128, 32, 128, 72, 0.08, 150, (10000.0, 32)), _dense(192)),
        _layer(_latent(3, 64, 16, 64, 64, 0.11, 70, (50000.0, 16), kv_from=0), _dense(192)),
    ],
}
KAKIPEL = {
    "architecture": "Kakipel", "vocab": 211, "width": 128, "norm": {"eps": 1e-6}, "initializer_range": 0.08, "loop": None,
    "layers": [kaki_layer(_mixer(3, 64, 16, 64, 64, 48, 0.11, 10000.0), DENSE(192)), kaki_layer(_mixer(2, 128, 48, 128, 96, 56, 0.08, 500.0), DENSE(192))],
}
PORTIONS = [70, 65, 130, 1, 64, 30, 73]
TOKENS = sum(PORTIONS)


@pytest.fixture(scope="module")
def kernels():
    from kvcache_b200.kernels.api import CudaKernels
    return CudaKernels(DEV)


def _folder(tmp_path, name):
    if name == "karorax":
        return make_karorax_folder(tmp_path, "F", dtype=torch.bfloat16, data=KARORAX)
    from kvcache_b200.config import config_from_dict
    from kvcache_b200.weights import write_random_model
    folder = os.path.join(str(tmp_path), "kaki_F")
    write_random_model(folder, config_from_dict(KAKIPEL), 0, torch.bfloat16)
    return folder


@pytest.mark.parametrize("name", ["karorax", "kakipel"])
def test_portions_that_start_anywhere(tmp_path, kernels, name):
    folder = _folder(tmp_path, name)
    runner = make_runner(folder, kernels, dtype="bfloat16", device=DEV, page_size=16, num_pages=96, max_tokens_per_step=TOKENS,
                         max_tokens_per_request=TOKENS + 16)
    plain = plain_karorax if name == "karorax" else plain_kakipel
    config, weights = plain.read_folder(folder)
    tokens = random_tokens(config["vocab"], TOKENS, 3)
    want = (plain.forward if name == "karorax" else plain.logits_of)(config, weights, tokens)
    spread = _spread(config, weights, tokens, want) if name == "karorax" else None
    for how, parts in (("whole", [TOKENS]), ("portions", PORTIONS)):
        before = kernels.launch_counts["attention_pairs_expanded"]
        got = replay_modes.portions(runner, tokens, parts)
        kernels.check_errors()
        expanded = sum(n >= 64 for n in parts) * len(config["layers"])
        assert kernels.launch_counts["attention_pairs_expanded"] - before == expanded, how
        if name == "karorax":
            assert_model_close(got, want, "bfloat16", how, spread)
        else:
            assert_close(got, want, 3e-2, how)


@pytest.mark.parametrize("name", ["karorax", "kakipel"])
def test_generation_with_and_without_graphs(tmp_path, kernels, name):
    """Prompts longer than a step, cut where the scheduler cuts them, then decoded: nothing raises, and every chosen token's logit is, by the
    plain implementation, the largest or within rounding of it."""
    from kvcache_b200 import LLM, SamplingParams
    folder = _folder(tmp_path, name)
    prompts = [random_tokens(211, n, 40 + n) for n in (400, 333, 90, 351)]
    for graphs in (False, True):
        llm = LLM(folder, kernels=kernels, dtype="bfloat16", device=DEV, page_size=16, num_pages=200, max_running=2, max_tokens_per_step=200,
                  use_graphs=graphs)
        llm.core.runner.graph_after_sightings = 2
        outs = llm.generate(prompts, SamplingParams(max_new_tokens=10, ignore_eos=True))
        assert llm.core.cache.used_pages() == 0
        for prompt, out in zip(prompts, outs):
            assert len(out) == 10
            if name == "kakipel":                                    # (the other one's plain implementation takes seconds a prompt)
                config, weights = plain_kakipel.read_folder(folder)
                rows = plain_kakipel.logits_of(config, weights, prompt + out[:-1])[len(prompt) - 1:]
                best = rows.max(dim=1).values
                assert (rows[torch.arange(10), torch.tensor(out)] >= best - 2 * 3e-2 * rows.abs().max(dim=1).values).all()


@pytest.mark.parametrize("name", ["karorax", "kakipel"])
def test_timing_names_the_expanded_attention(tmp_path, kernels, name):
    """With timing on, a portion's report holds the operator with its launches, bytes and multiply-adds, and a decoded token's does not."""
    from kvcache_b200.engine.runner import StepEntry
    runner = make_runner(_folder(tmp_path, name), kernels, dtype="bfloat16", device=DEV, page_size=16, num_pages=96, max_tokens_per_step=256)
    slot = runner.cache.admit()
    tokens = random_tokens(211, 201, 4)
    reports = []
    for part in (tokens[:200], tokens[200:]):
        kernels.start_timing(hold_ms=0.0)
        runner.step([StepEntry(slot, part, [len(part) - 1])])
        reports.append(kernels.stop_timing())
    runner.cache.release(slot)
    kernels.check_errors()
    layers = KARORAX["layers"] if name == "karorax" else KAKIPEL["layers"]
    entry = reports[0]["latent_expanded_attention"]
    assert entry["calls"] == len(layers) and entry["launches"] == 3 * len(layers) and "latent_attention" not in reports[0]
    assert reports[1]["latent_attention"]["calls"] == len(layers) and "latent_expanded_attention" not in reports[1]
    flops = nbytes = 0
    for m in (layer["mixer"] for layer in layers):
        window, H, dim, rot, rank = m.get("mask", {}).get("size"), m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
        seen = sum(min(p + 1, window or p + 1) for p in range(200))
        flops += 2 * 200 * 2 * H * dim * rank + 2 * H * (2 * dim + rot) * seen
        nbytes += 2 * (200 * (rank + rot) + 2 * H * dim * rank + 200 * H * (dim + rot + (1 if name == "karorax" else dim)) + 200 * H * dim)
    assert entry["flops"] == flops and entry["bytes"] == nbytes

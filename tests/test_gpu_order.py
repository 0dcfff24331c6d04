"""Shapes so small that CTAs of the streaming decode kernel stand idle in phases of a layer, over many layers.

Tolerance: none.  With at most 256 positions to a cache tile a context of 60 is one tile, which one CTA goes through, and every sum of a
projection is one CTA's; how many CTAs there are moves no sum, and the results of a few, all at work in every phase, are those of all."""

import pytest
import torch

from megabake_b200.synth import new_kv_state, synth_ids, synth_normal, synth_weights, tiny_config
from test_gpu_parity import make_kernel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,heads,kv_heads,intermediate", [(64, 1, 1, 64), (128, 2, 1, 256), (256, 4, 2, 512), (320, 5, 5, 192)])
@pytest.mark.parametrize("batch", [1, 4, 8, 16, 32])
def test_streaming_decode_of_small_shapes_with_many_layers(hidden, heads, kv_heads, intermediate, batch):
    device = torch.device("cuda:0")
    config = tiny_config(hidden=hidden, layers=12, q_heads=heads, kv_heads=kv_heads, intermediate=intermediate, vocab=4096)
    weights = synth_weights(config, seed=41, norm_std=0.1, device=device)
    results = []
    for sm_limit in (2, 0):
        kernel = make_kernel(config, weights, device, max_tokens=batch, max_positions=96, sm_limit=sm_limit)
        keys, values, lengths = new_kv_state(config, batch, 96, device)
        for layer in range(config.layers):
            for name, caches in (("k", keys), ("v", values)):
                caches[layer].copy_(synth_normal(tuple(caches[layer].shape), seed=41, name=f"{name}{layer}", std=0.5, device=device))
            lengths[layer].fill_(30)
        ids = synth_ids(batch, config.vocab, seed=41).view(batch, 1).to(device)
        logits = []
        for step in range(12):
            logits.append(kernel.decode(ids, torch.full((batch, 1), 30 + step, device=device), keys, values, lengths))
            kernel.check()
        results.append((torch.stack(logits), torch.stack(keys), torch.stack(values)))
    for few, every in zip(*results):
        assert torch.equal(few, every)

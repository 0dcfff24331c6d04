"""RoPE tables that begin at any element: decode takes them, a prompt refuses what its loads cannot take.

Tolerance: the one of the parity tests, 2e-2 absolute + 1e-2 relative: the two kernels and the two forms of decode attention that a table's
place chooses between round to bf16 at the same places or one rounding apart, in two layers."""

import pytest
import torch

from conftest import assert_parity
from megabake_b200.diagnostics import CompilerError
from megabake_b200.synth import new_kv_state, rope_tables, synth_ids, synth_normal, synth_weights, tiny_config
from test_gpu_parity import make_kernel

pytestmark = pytest.mark.gpu
DEVICE = torch.device("cuda:0")


def _tables(config, positions, offset):
    moved = []
    for table in rope_tables(config, positions, device=DEVICE):
        room = torch.zeros(table.numel() + 64, dtype=table.dtype, device=DEVICE)
        view = room[offset:offset + table.numel()].view(table.shape)
        moved.append(view.copy_(table))
    return tuple(moved)


def _step(config, weights, batch, context, offset, engine):
    kernel = make_kernel(config, weights, DEVICE, max_tokens=batch, max_positions=context + 4, engine=engine,
                         tables=_tables(config, context + 4, offset))
    keys, values, lengths = new_kv_state(config, batch, context + 4, DEVICE)
    for layer in range(config.layers):
        for name, caches in (("k", keys), ("v", values)):
            caches[layer].copy_(synth_normal(tuple(caches[layer].shape), seed=51, name=f"{name}{layer}", std=0.5, device=DEVICE))
        lengths[layer].fill_(context)
    ids = synth_ids(batch, config.vocab, seed=51).view(batch, 1).to(DEVICE)
    logits = kernel.decode(ids, torch.full((batch, 1), context, device=DEVICE), keys, values, lengths)
    kernel.check()
    return logits


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(4, 2, 64), (8, 2, 128)])
@pytest.mark.parametrize("batch,context", [(1, 20), (3, 300), (40, 1500)])
@pytest.mark.parametrize("engine", ["auto", "tcgen05"])
def test_decode_takes_tables_that_begin_at_any_element(heads, kv_heads, head_dim, batch, context, engine):
    config = tiny_config(hidden=512, q_heads=heads, kv_heads=kv_heads, head_dim=head_dim)
    weights = synth_weights(config, seed=51, norm_std=0.1, device=DEVICE)
    expected = _step(config, weights, batch, context, 0, engine)
    for offset in (1, 2, 4, 8):
        logits = _step(config, weights, batch, context, offset, engine)
        assert_parity(logits, expected, f"tables {offset} elements on")
        if offset == 8 or (offset > 1 and engine == "auto" and batch <= 32):  # the same kernel, the same form
            assert torch.equal(logits, expected)


def test_a_prompt_refuses_tables_off_16_bytes():
    config = tiny_config()
    weights = synth_weights(config, seed=51, norm_std=0.1, device=DEVICE)
    ids = synth_ids(20, config.vocab, seed=51).view(1, 20).to(DEVICE)
    results = {}
    for offset in (0, 1, 4, 8):
        kernel = make_kernel(config, weights, DEVICE, max_tokens=20, max_positions=32, tables=_tables(config, 32, offset))
        if offset in (1, 4):
            with pytest.raises(CompilerError, match="16-byte aligned"):
                kernel.prefill(ids)
        else:
            results[offset] = kernel.prefill(ids)
            kernel.check()
    assert torch.equal(results[0], results[8])

"""The sizes at which the kernels' own splits have their edges, against the oracle.

Tolerance: the one of the parity tests, 2e-2 absolute + 1e-2 relative.  Both sides round to bf16 (2^-9 relative) at the
same places or one rounding apart, a few such roundings meet in an output of these one- and two-layer shapes, and the
values are of order one: half of the bound is what the longest chain here can reach.
"""

import pytest
import torch

from conftest import assert_parity
from megabake_b200.synth import new_kv_state, rope_tables, synth_ids, synth_normal, synth_weights, tiny_config
from test_gpu_parity import make_kernel, oracle_decode_compare

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def device():
    return torch.device("cuda:0")


@pytest.mark.parametrize("batch,heads,kv_heads,head_dim,context,vocab", [
    (1, 4, 4, 64, 0, 250), (1, 8, 2, 64, 255, 333), (1, 9, 3, 64, 256, 512), (1, 7, 1, 128, 257, 512),  # one token: its own kernel class
    (4, 8, 8, 64, 511, 512), (5, 9, 3, 64, 64, 250),    # last size of the second class, first of the third
    (8, 4, 2, 128, 129, 512), (9, 8, 2, 64, 300, 333),  # one MMA tile of tokens, two
    (16, 4, 4, 128, 40, 512), (17, 8, 8, 64, 200, 250), (32, 14, 2, 64, 70, 512), (33, 4, 2, 64, 90, 512),  # two, four, past the kernel
])
def test_streaming_decode_at_class_and_tile_edges(device, batch, heads, kv_heads, head_dim, context, vocab):
    config = tiny_config(hidden=512, q_heads=heads, kv_heads=kv_heads, head_dim=head_dim, intermediate=768, vocab=vocab)
    oracle_decode_compare(config, device, batch=batch, capacity=context + 2, prefill=context, steps=2)


@pytest.mark.parametrize("batch,context", [(batch, context) for batch in (16, 32) for context in (0, 15, 16, 30, 31)])
def test_streaming_decode_with_a_context_of_one_tile_to_a_warp(device, batch, context):
    """Eight heads to a tile of 32 positions: every warp has its head's whole context, and none waits for another.  From 32
    positions on there is a second tile."""
    config = tiny_config(hidden=512, q_heads=32, kv_heads=32, head_dim=64, intermediate=768, vocab=512)
    oracle_decode_compare(config, device, batch=batch, capacity=context + 3, prefill=context, steps=3)


@pytest.mark.parametrize("batch,heads,kv_heads,head_dim", [(1, 9, 3, 64), (1, 4, 4, 64), (3, 14, 2, 64), (8, 8, 8, 64), (2, 8, 2, 128), (16, 32, 32, 64)])
@pytest.mark.parametrize("context", [0, 14, 15, 16, 31, 47, 48, 127, 128, 240, 256, 271])
def test_streaming_decode_reads_nothing_behind_the_new_position(device, batch, heads, kv_heads, head_dim, context):
    """Blocks of 16 positions behind the new one are left out, its own block is cleared behind it: whatever the caches hold there, not
    numbers included, the result is the one beside zeros, in every bit."""
    config = tiny_config(hidden=512, q_heads=heads, kv_heads=kv_heads, head_dim=head_dim, intermediate=768)
    capacity = context + 300
    kernel = make_kernel(config, synth_weights(config, seed=21, norm_std=0.1, device=device), device, max_tokens=batch, max_positions=capacity)
    ids = synth_ids(batch, config.vocab, seed=21).view(batch, 1).to(device)
    positions = torch.full((batch, 1), context, dtype=torch.int64, device=device)
    results = []
    for behind in (0.0, float("nan"), float("inf")):
        keys, values, lengths = new_kv_state(config, batch, capacity, device)
        for layer in range(config.layers):
            for name, caches in (("k", keys), ("v", values)):
                caches[layer].copy_(synth_normal(tuple(caches[layer].shape), seed=21, name=f"{name}{layer}", std=0.5, device=device))
                caches[layer][:, context:] = behind
            lengths[layer].fill_(context)
        results.append(kernel.decode(ids, positions, keys, values, lengths))
        kernel.check()
    assert bool(torch.isfinite(results[0]).all())
    assert torch.equal(results[0], results[1]) and torch.equal(results[0], results[2])


@pytest.mark.parametrize("lengths_now,sm_limit", [
    ([1000] * 28 + [10] * 4, 0), ([10] * 7 + [4000] * 9, 0), ([8000] * 6 + [10] * 6, 0),  # 17, 22 and 42 parts in one CTA
    ([40] * 32, 4),                                                                       # 32 of equal lengths: few CTAs
])
def test_streaming_decode_with_more_parts_than_a_list_holds(device, lengths_now, sm_limit):
    """Long sequences make the runs long, and a run through short ones crosses a head group per tile.  Every sequence must
    come out as if it had been decoded alone."""
    from oracle import decoder_oracle as oracle

    config = tiny_config(hidden=512, q_heads=32, kv_heads=32, head_dim=64, intermediate=768)
    batch, capacity = len(lengths_now), max(lengths_now) + 2
    weights = synth_weights(config, seed=16, norm_std=0.1, device=device)
    kernel = make_kernel(config, weights, device, max_tokens=batch, max_positions=capacity, sm_limit=sm_limit)
    tables = rope_tables(config, capacity, device=device)
    keys, values, _ = new_kv_state(config, batch, capacity, device)
    for layer in range(config.layers):
        for name, caches in (("k", keys), ("v", values)):
            caches[layer].copy_(synth_normal(tuple(caches[layer].shape), seed=16, name=f"{name}{layer}", std=0.5, device=device))
    lengths = [torch.tensor(lengths_now, dtype=torch.int32, device=device) for _ in range(config.layers)]
    alone = [([k[row:row + 1].clone() for k in keys], [v[row:row + 1].clone() for v in values],
              [torch.full((1,), filled, dtype=torch.int32, device=device) for _ in range(config.layers)])
             for row, filled in enumerate(lengths_now)]
    ids = synth_ids(batch, config.vocab, seed=16).view(batch, 1).to(device)
    for step in range(2):
        positions = torch.tensor([[n + step] for n in lengths_now], dtype=torch.int64, device=device)
        logits = kernel.decode_ragged(ids, positions, keys, values, lengths)
        kernel.check()
        with torch.no_grad():
            expected = torch.cat([oracle.decode_step(config, weights, tables, ids[row:row + 1], positions[row:row + 1], *alone[row])
                                  for row in range(batch)])
        assert_parity(logits, expected, f"logits at step {step}")
    for row, filled in enumerate(lengths_now):
        assert_parity(keys[-1][row, :filled + 2], alone[row][0][-1][0, :filled + 2], f"sequence {row} key cache")
        assert_parity(values[-1][row, :filled + 2], alone[row][1][-1][0, :filled + 2], f"sequence {row} value cache")


@pytest.mark.parametrize("kv_heads,head_dim,context", [(40, 64, 300), (40, 64, 319), (20, 128, 258)])
def test_tensor_engine_attention_with_two_units_to_a_block(device, kv_heads, head_dim, context):
    """More (sequence, head group) units than SMs: the second unit's cache stream starts before the first one ends."""
    config = tiny_config(hidden=256, q_heads=kv_heads, kv_heads=kv_heads, head_dim=head_dim)
    oracle_decode_compare(config, device, batch=32, capacity=context + 2, prefill=context, steps=2, engine="tcgen05")


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(8, 1, 64), (3, 3, 64), (8, 2, 128), (16, 8, 64)])
@pytest.mark.parametrize("context", [0, 63, 130, 300, 700, 1023])
def test_tensor_engine_attention_with_any_number_of_chunks(device, heads, kv_heads, head_dim, context):
    """A context in 1 to 16 chunks of up to 64 positions: their statistics and sums come four chunks and four columns at a time, whatever is
    there of them."""
    config = tiny_config(hidden=256, q_heads=heads, kv_heads=kv_heads, head_dim=head_dim)
    oracle_decode_compare(config, device, batch=1, capacity=context + 3, prefill=context, steps=2, engine="tcgen05")


@pytest.mark.parametrize("heads,kv_heads,head_dim,batch,context", [(16, 4, 64, 80, 1300), (8, 2, 128, 120, 1290), (8, 1, 64, 120, 2600)])
def test_tensor_engine_attention_of_more_units_than_ctas(device, heads, kv_heads, head_dim, batch, context):
    """Chunks that have to be cut for their scores' room, two or three to a CTA one behind the other: a sequence's chunks are summed
    at the end of the phase by the CTA that had the first of them, some CTAs for several sequences and some for none."""
    config = tiny_config(hidden=256, q_heads=heads, kv_heads=kv_heads, head_dim=head_dim)
    oracle_decode_compare(config, device, batch=batch, capacity=context + 3, prefill=context, steps=2, engine="tcgen05")


@pytest.mark.parametrize("tokens", [16, 17, 64, 65, 128, 129, 256, 257, 385, 513])
@pytest.mark.parametrize("head_dim", [64, 128])
def test_prompts_at_token_tile_edges(device, tokens, head_dim):
    """One token tile (16 to 128), then a unit per token tile with tables for two, three and four or more."""
    from oracle import decoder_oracle as oracle

    config = tiny_config(hidden=512, q_heads=6, kv_heads=2, head_dim=head_dim, intermediate=832, rope_style="hf")
    weights = synth_weights(config, seed=12, norm_std=0.1, device=device)
    kernel = make_kernel(config, weights, device, max_tokens=tokens, max_positions=tokens)
    ids = synth_ids(tokens, config.vocab, seed=12).view(1, tokens).to(device)
    positions = torch.arange(tokens, device=device).view(1, tokens)
    with torch.no_grad():
        expected = oracle.prefill(config, weights, rope_tables(config, tokens, device=device), ids, positions,
                                  oracle.causal_mask(1, tokens).to(device))
    logits = kernel.prefill(ids)
    kernel.check()
    assert_parity(logits, expected, f"prompt of {tokens}")


@pytest.mark.parametrize("heads,kv_heads,head_dim,intermediate", [(9, 3, 64, 832), (3, 1, 64, 64), (5, 5, 128, 448), (2, 1, 128, 1088)])
@pytest.mark.parametrize("tokens", [1, 2, 31, 33, 63, 66, 127])
def test_short_prompts_whose_tiles_end_in_either_half(device, heads, kv_heads, head_dim, intermediate, tokens):
    """Up to 128 tokens, projections on pairs: half of the tokens and half of a tile's weight rows to each CTA.  Odd numbers of heads and
    narrow matrices end in the first half or in the second; one token leaves the second CTA without any."""
    from oracle import decoder_oracle as oracle

    config = tiny_config(hidden=320, q_heads=heads, kv_heads=kv_heads, head_dim=head_dim, intermediate=intermediate, vocab=1003, qkv_bias=True)
    weights = synth_weights(config, seed=31, norm_std=0.1, device=device)
    kernel = make_kernel(config, weights, device, max_tokens=tokens, max_positions=max(tokens, 16))
    ids = synth_ids(tokens, config.vocab, seed=31).view(1, tokens).to(device)
    positions = torch.arange(tokens, device=device).view(1, tokens)
    with torch.no_grad():
        expected = oracle.prefill(config, weights, rope_tables(config, max(tokens, 16), device=device), ids, positions,
                                  oracle.causal_mask(1, tokens).to(device))
    assert_parity(kernel.prefill(ids), expected, f"prompt of {tokens}")
    kernel.check()


@pytest.mark.parametrize("batch,sequence", [(1, 1), (3, 7), (2, 33), (5, 25), (3, 61), (4, 129)])
@pytest.mark.parametrize("head_dim", [64, 128])
def test_prompts_with_biases_masks_and_buffers_on_any_element(device, batch, sequence, head_dim):
    """Every kind of launch (tiles of 64 and 128 tokens, one and more tiles of a CTA pair) with several sequences, a mask,
    projections with biases that begin at an odd element, a vocabulary that ends inside a tile and logits at an odd element."""
    from megabake_b200 import _native
    from oracle import decoder_oracle as oracle

    config = tiny_config(hidden=192, q_heads=6, kv_heads=2, head_dim=head_dim, intermediate=320, vocab=333, rope_style="hf",
                         qkv_bias=True)
    weights = dict(synth_weights(config, seed=21, norm_std=0.1, device=device))
    for name, tensor in weights.items():
        if name.endswith("proj.bias"):
            off = torch.empty(tensor.numel() + 1, dtype=tensor.dtype, device=device)[1:]
            weights[name] = off.copy_(tensor)
    tokens = batch * sequence
    kernel = make_kernel(config, weights, device, max_tokens=tokens, max_positions=max(sequence, 16))
    ids = synth_ids(tokens, config.vocab, seed=22).view(batch, sequence).to(device)
    positions = torch.arange(sequence, device=device).expand(batch, sequence).contiguous()
    mask = oracle.causal_mask(batch, sequence).to(device).contiguous()
    mask[:, :, :, : sequence // 3] = torch.finfo(torch.bfloat16).min
    mask[:, :, :, 0] = 0.0  # every row sees something
    with torch.no_grad():
        expected = oracle.prefill(config, weights, rope_tables(config, max(sequence, 16), device=device), ids, positions, mask)
    assert_parity(kernel.prefill(ids, positions, mask), expected, "logits")
    store = torch.empty(tokens * config.vocab + 2, dtype=torch.bfloat16, device=device).fill_(7.0)
    _native.check("mk_prefill", kernel.lib.mk_prefill(kernel._handle, ids.data_ptr(), positions.data_ptr(), mask.data_ptr(), batch,
                                                      sequence, store[1:].data_ptr(), torch.cuda.current_stream().cuda_stream))
    kernel.check()
    assert_parity(store[1:-1].view(batch, sequence, -1), expected, "logits at an odd element")
    assert store[0].item() == 7.0 and store[-1].item() == 7.0


@pytest.mark.parametrize("tokens", [40, 200])
def test_a_refused_prompt_is_all_nan_and_the_next_one_is_not(device, tokens):
    config = tiny_config(hidden=192, intermediate=320, rope_style="hf")
    weights = synth_weights(config, seed=23, device=device)
    kernel = make_kernel(config, weights, device, max_tokens=tokens, max_positions=tokens)
    ids = synth_ids(tokens, config.vocab, seed=23).view(1, tokens).to(device)
    fine = kernel.prefill(ids)
    kernel.check()
    for bad_ids, bad_position in ((config.vocab, tokens - 1), (-1, 0), (0, tokens)):
        wrong, positions = ids.clone(), torch.arange(tokens, device=device).view(1, tokens).clone()
        wrong[0, tokens // 2] = bad_ids
        positions[0, -1] = bad_position
        logits = kernel.prefill(wrong, positions)
        assert kernel.status()["status"] == "BAD_INDEX" and torch.isnan(logits).all()
        assert torch.equal(kernel.prefill(ids), fine)
        kernel.check()


@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("keys", [64, 65, 191, 256, 333])
@pytest.mark.parametrize("offset", [2, 8])
def test_prompt_attention_op_with_operands_on_any_word_and_infinite_masks(device, head_dim, keys, offset):
    """Queries off the 16-byte grid, masks that begin at an odd element, rows whose first tiles are all -inf, rows that see
    nothing: zeros."""
    from oracle import decoder_oracle as oracle

    heads, kv_heads, batch = 6, 2, 2
    query, key, value = _tensors(device, batch, keys, keys, heads, kv_heads, head_dim)
    moved = torch.empty(query.numel() + offset, dtype=query.dtype, device=device)[offset:].view(query.shape).copy_(query)
    store = torch.zeros(batch * keys * keys + 1, dtype=torch.bfloat16, device=device)
    mask = store[1:].view(batch, 1, keys, keys)
    rows, columns = torch.arange(keys, device=device).view(-1, 1), torch.arange(keys, device=device)
    mask.masked_fill_((columns > rows) | (columns < rows - 20), -torch.inf)
    out = torch.ops.megabake.attention(moved, key, value, mask, head_dim ** -0.5)
    assert_parity(out, oracle.attention(query, key, value, mask, head_dim ** -0.5), f"attention over {keys}")
    mask[:, :, 5] = -torch.inf
    again = torch.ops.megabake.attention(moved, key, value, mask, head_dim ** -0.5)
    assert (again[:, 5] == 0).all() and torch.equal(again[:, 6:], out[:, 6:])


@pytest.mark.parametrize("keys", [40, 200])
def test_prompt_attention_with_queries_at_an_odd_element(device, keys):
    """The ops take them (a copy is attended), the C entry point refuses them and such outputs: the kernels read and write pairs."""
    from megabake_b200 import _native
    from megabake_b200.runtime import AttentionKernels

    query, key, value = _tensors(device, 2, keys, keys, 6, 2, 64)
    odd = torch.empty(query.numel() + 1, dtype=query.dtype, device=device)[1:].view(query.shape).copy_(query)
    expected = torch.ops.megabake.attention(query, key, value, None, 0.125)
    assert torch.equal(torch.ops.megabake.attention(odd, key, value, None, 0.125), expected)
    with torch.inference_mode():
        assert torch.equal(torch.ops.megabake.attention(odd, key, value, None, 0.125), expected)
    kernels = AttentionKernels.for_shape(6, 2, 64, 2 * keys, device)
    out = torch.full((expected.numel() + 1,), 7.0, dtype=torch.bfloat16, device=device)
    for q, result in ((odd, out), (query, out[1:])):
        code = kernels.lib.mk_attention(kernels._handle, q.data_ptr(), key.data_ptr(), value.data_ptr(), None, 0.125, 2, keys, keys,
                                        result.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert code == _native.MK_ERR_ALIGNMENT
    assert (out == 7.0).all()


@pytest.mark.parametrize("sm_limit", [1, 7])
@pytest.mark.parametrize("tokens", [50, 300])
def test_prompts_on_few_sms(device, sm_limit, tokens):
    """Many units to a CTA: both accumulator buffers and every slot of the pipeline come around several times."""
    from oracle import decoder_oracle as oracle

    config = tiny_config(hidden=512, q_heads=6, kv_heads=2, intermediate=832, vocab=1003, rope_style="hf")
    weights = synth_weights(config, seed=24, norm_std=0.1, device=device)
    kernel = make_kernel(config, weights, device, max_tokens=tokens, max_positions=tokens, sm_limit=sm_limit)
    ids = synth_ids(tokens, config.vocab, seed=24).view(1, tokens).to(device)
    positions = torch.arange(tokens, device=device).view(1, tokens)
    with torch.no_grad():
        expected = oracle.prefill(config, weights, rope_tables(config, tokens, device=device), ids, positions,
                                  oracle.causal_mask(1, tokens).to(device))
    assert_parity(kernel.prefill(ids), expected, f"prompt of {tokens} on {sm_limit}")
    kernel.check()


def test_gates_beyond_the_straight_line_of_the_silu(device):
    """Gates past +-80 take the epilogue's plain division, their neighbours in a token's column the corrected quotient."""
    from oracle import decoder_oracle as oracle

    config = tiny_config(hidden=512, q_heads=6, kv_heads=2, intermediate=832, rope_style="hf")
    weights = dict(synth_weights(config, seed=15, norm_std=0.1, device=device))
    for layer in range(config.layers):
        for name, factor in (("gate", 64.0), ("up", 1 / 64.0)):  # powers of two: the products only change their exponents
            key = f"model.layers.{layer}.mlp.{name}_proj.weight"
            weights[key] = (weights[key] * factor).contiguous()
    tokens = 40
    kernel = make_kernel(config, weights, device, max_tokens=tokens, max_positions=tokens)
    ids = synth_ids(tokens, config.vocab, seed=15).view(1, tokens).to(device)
    positions = torch.arange(tokens, device=device).view(1, tokens)
    with torch.no_grad():
        expected = oracle.prefill(config, weights, rope_tables(config, tokens, device=device), ids, positions,
                                  oracle.causal_mask(1, tokens).to(device))
    assert_parity(kernel.prefill(ids), expected, "prompt with large gates")
    kernel.check()


def _tensors(device, batch, queries, keys, heads, kv_heads, head_dim):
    return [synth_normal((batch, n, h, head_dim), seed=13, name=name, std=1.0, device=device)
            for name, n, h in (("q", queries, heads), ("k", keys, kv_heads), ("v", keys, kv_heads))]


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(9, 3, 64), (8, 2, 128)])
@pytest.mark.parametrize("queries,keys", [(1, 1), (1, 65), (63, 63), (64, 64), (65, 65), (130, 33), (200, 449)])
@pytest.mark.parametrize("masked", [False, True])
def test_prompt_attention_op_at_block_and_tile_edges(device, heads, kv_heads, head_dim, queries, keys, masked):
    """Ragged query blocks and key tiles, odd key counts (mask rows off the 4-byte grid), rows that begin with whole tiles of
    the lowest finite mask value."""
    from oracle import decoder_oracle as oracle

    query, key, value = _tensors(device, 2, queries, keys, heads, kv_heads, head_dim)
    mask = None
    if masked:
        mask = torch.zeros((2, 1, queries, keys), dtype=torch.bfloat16, device=device)
        hidden = torch.arange(keys, device=device) < torch.arange(queries, device=device).view(-1, 1).clamp(max=keys - 1)
        mask[:, 0].masked_fill_(hidden, torch.finfo(torch.bfloat16).min)
    out = torch.ops.megabake.attention(query, key, value, mask, head_dim ** -0.5)
    expected = oracle.attention(query, key, value, mask, head_dim ** -0.5)
    assert_parity(out, expected, f"attention {queries} x {keys}")


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(9, 3, 64), (14, 2, 64), (11, 11, 64), (32, 32, 64), (32, 8, 128)])
@pytest.mark.parametrize("batch,context", [(1, 0), (3, 15), (1, 16), (2, 17), (16, 63), (2, 700)])
def test_decode_attention_op_at_tile_and_run_edges(device, heads, kv_heads, head_dim, batch, context):
    """The new position first, last and alone in a tile of 16, runs of positions without any; cache rows past the valid
    length hold NaN, which must not reach the result."""
    from oracle import decoder_oracle as oracle

    capacity = context + 5
    query, key, value = _tensors(device, batch, 1, 1, heads, kv_heads, head_dim)
    caches = [synth_normal((batch, capacity, kv_heads, head_dim), seed=14, name=name, std=1.0, device=device) for name in ("kc", "vc")]
    for cache in caches:
        cache[:, context:] = float("nan")
    mine, ref = [c.clone() for c in caches], [c.clone() for c in caches]
    length, ref_length = (torch.full((1,), context, dtype=torch.int32, device=device) for _ in range(2))
    out = torch.ops.megabake.kv_attention(query, key, value, mine[0], mine[1], length)
    expected = oracle.kv_attention(query, key, value, ref[0], ref[1], ref_length)
    assert_parity(out, expected, f"kv_attention at {context}")
    assert int(length) == context + 1
    for a, b in zip(mine, ref):
        assert torch.equal(a[:, :context + 1], b[:, :context + 1]) and bool(torch.isnan(a[:, context + 1:].float()).all())


def _filled_decode(device, batch, context, heads=8, kv_heads=8, head_dim=64):
    """Query, key, value and the two caches of a decode attention call."""
    caches = [synth_normal((batch, context + 2, kv_heads, head_dim), seed=20, name=name, std=1.0, device=device) for name in ("kc", "vc")]
    return (*_tensors(device, batch, 1, 1, heads, kv_heads, head_dim), *caches)


@pytest.mark.parametrize("where", [0, 40, 700, 1023])
@pytest.mark.parametrize("spoilt", [float("nan"), float("inf")])
def test_decode_attention_op_shows_a_key_that_is_not_a_number(device, where, spoilt):
    """One spoilt key in a context of several parts: its heads' results are not numbers, wherever the context was cut."""
    query, key, value, key_cache, value_cache = _filled_decode(device, 2, 1024)
    query[:, 0, 3, 0] = 1.0
    key_cache[1, where, 3, 0] = spoilt
    out = torch.ops.megabake.kv_attention(query, key, value, key_cache, value_cache, torch.full((1,), 1024, dtype=torch.int32, device=device))
    bad = torch.isnan(out.float()).view(2, 8, 64)
    assert bool(bad[1, 3].all()) and int(bad.sum()) == 64


@pytest.mark.parametrize("hidden", [1, 16, 300, 1023])
def test_decode_attention_op_with_scores_of_minus_infinity(device, hidden):
    """Positions with a score of -inf weigh nothing, also where a warp, or a whole run of positions, has no others."""
    from oracle import decoder_oracle as oracle

    query, key, value, key_cache, value_cache = _filled_decode(device, 2, 1024, heads=14, kv_heads=2)
    query[..., 0] = 1.0
    key_cache[:, :hidden, :, 0] = float("-inf")
    caches = [key_cache.clone(), value_cache.clone()]
    length, ref_length = (torch.full((1,), 1024, dtype=torch.int32, device=device) for _ in range(2))
    out = torch.ops.megabake.kv_attention(query, key, value, key_cache, value_cache, length)
    assert_parity(out, oracle.kv_attention(query, key, value, *caches, ref_length), f"{hidden} positions of -inf")


@pytest.mark.parametrize("context", [0, 3, 15, 1000])
def test_decode_attention_op_with_an_infinite_new_value(device, context):
    """The positions that pad the last tile must not turn it into something that is not a number."""
    from oracle import decoder_oracle as oracle

    query, key, value, key_cache, value_cache = _filled_decode(device, 2, context)
    value[0, 0, 5, 7] = float("inf")
    caches = [key_cache.clone(), value_cache.clone()]
    length, ref_length = (torch.full((1,), context, dtype=torch.int32, device=device) for _ in range(2))
    out = torch.ops.megabake.kv_attention(query, key, value, key_cache, value_cache, length)
    expected = oracle.kv_attention(query, key, value, *caches, ref_length)
    infinite = torch.isinf(expected.float())
    assert int(infinite.sum()) == 1 and torch.equal(out[infinite], expected[infinite])
    assert_parity(out.masked_fill(infinite, 0.0), expected.masked_fill(infinite, 0.0), "the finite results")


@pytest.mark.parametrize("batch,context,hidden", [(1, 700, 400), (1, 700, 699), (16, 1100, 1000), (32, 70, 30), (2, 20, 17)])
def test_streaming_decode_with_scores_of_minus_infinity(device, batch, context, hidden):
    """The same in the streaming kernel: q is its bias (1 in every place, position 0 does not rotate), so that the cached keys
    decide which scores are -inf."""
    from oracle import decoder_oracle as oracle

    config = tiny_config(hidden=512, q_heads=16, kv_heads=16, intermediate=768, layers=1, qkv_bias=True)
    weights = dict(synth_weights(config, seed=19, norm_std=0.1, device=device))
    prefix = "model.layers.0.self_attn."
    weights[prefix + "q_proj.weight"] = torch.zeros_like(weights[prefix + "q_proj.weight"])
    weights[prefix + "q_proj.bias"] = torch.ones_like(weights[prefix + "q_proj.bias"])
    kernel = make_kernel(config, weights, device, max_tokens=batch, max_positions=16)
    keys, values, lengths = new_kv_state(config, batch, context + 2, device)
    keys[0].copy_(synth_normal(tuple(keys[0].shape), seed=19, name="k", std=0.3, device=device))
    values[0].copy_(synth_normal(tuple(values[0].shape), seed=19, name="v", std=1.0, device=device))
    keys[0][:, :hidden, :, 0] = float("-inf")
    lengths[0].fill_(context)
    ref = ([keys[0].clone()], [values[0].clone()], [lengths[0].clone()])
    ids = synth_ids(batch, config.vocab, seed=19).view(batch, 1).to(device)
    positions = torch.zeros((batch, 1), dtype=torch.int64, device=device)
    with torch.no_grad():
        expected = oracle.decode_step(config, weights, rope_tables(config, 16, device=device), ids, positions, *ref)
    assert bool(torch.isfinite(expected.float()).all())
    assert_parity(kernel.decode(ids, positions, keys, values, lengths), expected, f"{hidden} of {context} positions of -inf")
    kernel.check()


def _interleaved(device, call, rounds=40):
    """Decode attention calls of one head shape on two streams, whose launches may run in any order and side by side: small
    ones that leave room for the others."""
    from oracle import decoder_oracle as oracle

    heads, kv_heads, head_dim, capacity = 8, 8, 64, 1200
    streams, sides = [torch.cuda.Stream(device) for _ in range(2)], []
    for index, (batch, context) in enumerate(((1, 1100), (2, 37))):
        query, key, value = _tensors(device, batch, 1, 1, heads, kv_heads, head_dim)
        query, key, value = (t * (index + 1) for t in (query, key, value))
        caches = [synth_normal((batch, capacity, kv_heads, head_dim), seed=18 + index, name=name, std=1.0, device=device) for name in ("kc", "vc")]
        ref = [c.clone() for c in caches]
        expected = oracle.kv_attention(query, key, value, *ref, torch.full((1,), context, dtype=torch.int32, device=device))
        lengths = [torch.full((1,), context, dtype=torch.int32, device=device) for _ in range(rounds)]
        sides.append((query, key, value, caches, lengths, expected, context, []))
    torch.cuda.synchronize(device)
    for i in range(rounds):
        for stream, (query, key, value, caches, lengths, _, _, outs) in zip(streams, sides):
            with torch.cuda.stream(stream):
                outs.append(call(query, key, value, *caches, lengths[i]))
    torch.cuda.synchronize(device)
    for query, key, value, caches, lengths, expected, context, outs in sides:
        assert [int(n) for n in lengths] == [context + 1] * rounds
        for out in outs:
            assert_parity(out.view(expected.shape), expected, f"decode attention at {context} beside another stream's")


def test_decode_attention_op_on_two_streams(device):
    _interleaved(device, torch.ops.megabake.kv_attention)


def test_decode_attention_op_in_a_graph_beside_calls_on_the_capturing_stream(device):
    """A captured call's scratch is the graph's: replays beside eager calls on the stream that captured it."""
    from oracle import decoder_oracle as oracle

    query, key, value = _tensors(device, 1, 1, 1, 8, 8, 64)
    caches = [synth_normal((1, 1200, 8, 64), seed=21, name=name, std=1.0, device=device) for name in ("kc", "vc")]
    eager_caches = [c.clone() * 2 for c in caches]
    expected = oracle.kv_attention(query, key, value, *[c.clone() for c in caches], torch.full((1,), 1100, dtype=torch.int32, device=device))
    eager = oracle.kv_attention(query, key, value, *[c.clone() for c in eager_caches], torch.full((1,), 900, dtype=torch.int32, device=device))
    lengths, side, graph = [torch.zeros(1, dtype=torch.int32, device=device) for _ in range(2)], torch.cuda.Stream(device), torch.cuda.CUDAGraph()
    torch.cuda.synchronize(device)
    with torch.cuda.stream(side):
        lengths[1].fill_(900)
        torch.ops.megabake.kv_attention(query, key, value, *eager_caches, lengths[1])
    torch.cuda.synchronize(device)
    with torch.cuda.graph(graph, stream=side):
        lengths[0].fill_(1100)
        out = torch.ops.megabake.kv_attention(query, key, value, *caches, lengths[0])
    outs = []
    for _ in range(40):
        graph.replay()
        with torch.cuda.stream(side):
            lengths[1].fill_(900)
            outs.append(torch.ops.megabake.kv_attention(query, key, value, *eager_caches, lengths[1]))
    torch.cuda.synchronize(device)
    assert_parity(out.view(expected.shape), expected, "replayed decode attention")
    for each in outs:
        assert_parity(each.view(eager.shape), eager, "decode attention beside a replay")


def test_decode_attention_entry_point_with_the_handles_scratch_on_two_streams(device):
    from megabake_b200 import _native

    config = tiny_config(hidden=512, q_heads=8, kv_heads=8, head_dim=64)
    kernel = make_kernel(config, synth_weights(config, device=device), device, max_tokens=2, max_positions=16)

    def call(query, key, value, key_cache, value_cache, length):
        out = torch.empty((query.shape[0] * 8, 1, 64), dtype=torch.bfloat16, device=device)
        _native.check("mk_kv_attention", kernel.lib.mk_kv_attention(
            kernel._handle, query.data_ptr(), key.data_ptr(), value.data_ptr(), key_cache.data_ptr(), value_cache.data_ptr(),
            length.data_ptr(), query.shape[0], key_cache.shape[1], out.data_ptr(), torch.cuda.current_stream(device).cuda_stream))
        return out

    _interleaved(device, call)


def test_decode_attention_entry_point_refuses_scratch_that_is_too_small_or_misaligned(device):
    from megabake_b200 import _native

    config = tiny_config(hidden=512, q_heads=8, kv_heads=8, head_dim=64)
    kernel = make_kernel(config, synth_weights(config, device=device), device, max_tokens=2, max_positions=16)
    size = kernel.lib.mk_kv_attention_scratch_bytes(2, 8, 64)
    scratch = torch.empty(size + 16, dtype=torch.uint8, device=device)
    one = torch.zeros(2 * 16 * 512, dtype=torch.bfloat16, device=device)
    length = torch.zeros(1, dtype=torch.int32, device=device)

    def call(at, count):
        return kernel.lib.mk_kv_attention_scratch(kernel._handle, *[one.data_ptr()] * 5, length.data_ptr(), 2, 16, one.data_ptr(),
                                                  scratch.data_ptr() + at, count, None)

    assert call(0, size - 1) == _native.MK_ERR_WORKSPACE and call(8, size) == _native.MK_ERR_ALIGNMENT
    assert call(0, 0) == _native.MK_ERR_WORKSPACE and int(length) == 0


@pytest.mark.parametrize("batch", [1, 3, 4, 7, 12, 16, 29])
def test_streaming_decode_with_tiles_that_end_early(device, batch):
    """Rows that no tile height divides, a vocabulary that ends within a tile, and CTAs with several tiles: every warp of the
    epilogue has tokens, rows or copies that are not there."""
    config = tiny_config(hidden=320, q_heads=5, kv_heads=5, head_dim=64, intermediate=4992, vocab=5003)
    oracle_decode_compare(config, device, batch=batch, capacity=40, prefill=21, steps=3)


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(9, 3, 64), (8, 2, 128)])
@pytest.mark.parametrize("queries,keys", [(70, 72), (129, 128), (257, 200), (128, 456), (300, 704), (96, 200), (95, 1024), (15, 1032), (16, 1024)])
@pytest.mark.parametrize("offset", [0, 4, 1])
def test_prompt_attention_op_with_masks_that_come_in_tiles(device, heads, kv_heads, head_dim, queries, keys, offset):
    """Mask rows on 16-byte boundaries come by tiled copies where there are queries or positions enough, whose boxes end beyond the last position, query or sequence; the
    same mask elsewhere in memory comes row by row, with the same bits."""
    from oracle import decoder_oracle as oracle

    query, key, value = _tensors(device, 3, queries, keys, heads, kv_heads, head_dim)
    generator = torch.Generator(device=device).manual_seed(keys + queries)
    mask = torch.randn((3, 1, queries, keys), device=device, generator=generator).to(torch.bfloat16)
    mask[:, 0, :, 1:].masked_fill_(torch.rand((3, queries, keys - 1), device=device, generator=generator) < 0.4, torch.finfo(torch.bfloat16).min)
    moved = torch.empty(mask.numel() + offset, dtype=torch.bfloat16, device=device)[offset:].view(mask.shape)
    moved.copy_(mask)
    out = torch.ops.megabake.attention(query, key, value, moved, head_dim ** -0.5)
    assert_parity(out, oracle.attention(query, key, value, mask, head_dim ** -0.5), f"attention {queries} x {keys}")
    if offset:  # the other route
        assert torch.equal(out, torch.ops.megabake.attention(query, key, value, mask, head_dim ** -0.5))


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(9, 3, 64), (8, 2, 128)])
@pytest.mark.parametrize("queries,keys", [(96, 257), (128, 259), (129, 321), (200, 194), (257, 262), (300, 327), (64, 323), (33, 641), (256, 1020)])
@pytest.mark.parametrize("batch", [1, 3])
def test_prompt_attention_op_with_masks_whose_rows_begin_anywhere(device, heads, kv_heads, head_dim, queries, keys, batch):
    """Every residue of the row length modulo eight: copies of every eighth row, whose boxes begin before a row's first element and end beyond
    the last position, query or sequence.  The same mask at an odd element comes with loads, and with the same bits."""
    from oracle import decoder_oracle as oracle

    query, key, value = _tensors(device, batch, queries, keys, heads, kv_heads, head_dim)
    generator = torch.Generator(device=device).manual_seed(keys + queries)
    mask = torch.randn((batch, 1, queries, keys), device=device, generator=generator).to(torch.bfloat16)
    mask[:, 0, :, 1:].masked_fill_(torch.rand((batch, queries, keys - 1), device=device, generator=generator) < 0.4, float("-inf"))
    out = torch.ops.megabake.attention(query, key, value, mask, head_dim ** -0.5)
    assert_parity(out, oracle.attention(query, key, value, mask, head_dim ** -0.5), f"attention {queries} x {keys}")
    moved = torch.empty(mask.numel() + 1, dtype=torch.bfloat16, device=device)[1:].view(mask.shape).copy_(mask)
    assert torch.equal(out, torch.ops.megabake.attention(query, key, value, moved, head_dim ** -0.5))


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(6, 2, 64), (6, 2, 128)])
@pytest.mark.parametrize("keys", [456, 704, 701])
def test_prompt_attention_with_a_mask_and_several_units_to_a_block(device, heads, kv_heads, head_dim, keys):
    """On five SMs a block goes on from unit to unit: the ring of tiles carries over, and the exchange at a unit's end lies where the
    next one's queries, probabilities and (head size 128) first tile come.  701: masks off 16 bytes, copies of every eighth row."""
    from oracle import decoder_oracle as oracle

    query, key, value = _tensors(device, 2, 700, keys, heads, kv_heads, head_dim)
    mask = torch.randn((2, 1, 700, keys), device=device, generator=torch.Generator(device=device).manual_seed(keys)).to(torch.bfloat16)
    config = tiny_config(q_heads=heads, kv_heads=kv_heads, head_dim=head_dim, hidden=512)
    weights = synth_weights(config, seed=19, device=device)
    few, all_sms = (make_kernel(config, weights, device, max_tokens=16, max_positions=16, sm_limit=limit) for limit in (5, 0))
    out = few.attention(query, key, value, mask, head_dim ** -0.5)
    few.check()
    assert torch.equal(out, all_sms.attention(query, key, value, mask, head_dim ** -0.5))
    assert_parity(out, oracle.attention(query, key, value, mask, head_dim ** -0.5), f"attention 700 x {keys} on five SMs")


def test_streaming_decode_of_changing_batches_on_one_handle(device):
    """Launches of every plan and token class share the hand-over buffers, the barrier's count and the reset at a launch's end: each
    gives the bits of a handle that was never used."""
    config = tiny_config(hidden=576, q_heads=9, kv_heads=3, head_dim=64, intermediate=1536, layers=4)
    weights = synth_weights(config, seed=23, norm_std=0.1, device=device)
    kernel = make_kernel(config, weights, device, max_tokens=32, max_positions=80)
    for turn, batch in enumerate((1, 16, 3, 32, 8, 1, 12, 9, 5, 17, 2)):
        ids = synth_ids(batch, config.vocab, seed=turn).view(batch, 1).to(device)
        positions = torch.full((batch, 1), 70, dtype=torch.int64, device=device)
        results = []
        for used in (kernel, make_kernel(config, weights, device, max_tokens=32, max_positions=80)):
            keys, values, lengths = new_kv_state(config, batch, 80, device)
            for layer in range(config.layers):
                for name, cache in (("k", keys[layer]), ("v", values[layer])):
                    cache.copy_(synth_normal(tuple(cache.shape), seed=23, name=f"{name}{layer}", std=0.5, device=device))
                lengths[layer].fill_(70)
            tokens, logits = used.decode_steps(ids.clone(), positions.clone(), keys, values, lengths, steps=3, return_logits=True)
            used.check()
            results.append([tokens, logits, *keys, *values, *lengths])
        assert all(torch.equal(a, b) for a, b in zip(*results)), f"launch {turn}, batch {batch}"


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(9, 3, 64), (8, 2, 128)])
@pytest.mark.parametrize("queries,keys,masked", [(128, 512, True), (200, 449, False), (257, 200, True)])
def test_prompt_attention_op_gives_a_column_the_same_bits_in_either_half(device, heads, kv_heads, head_dim, queries, keys, masked):
    """Two groups of warps finish half of the columns each: with the halves of the values exchanged, those of the results are, bit
    by bit."""
    query, key, value = _tensors(device, 2, queries, keys, heads, kv_heads, head_dim)
    mask = torch.randn((2, 1, queries, keys), device=device, generator=torch.Generator(device=device).manual_seed(3)).to(torch.bfloat16) if masked else None
    out = torch.ops.megabake.attention(query, key, value, mask, head_dim ** -0.5)
    moved = torch.ops.megabake.attention(query, key, value.roll(head_dim // 2, -1), mask, head_dim ** -0.5)
    assert torch.equal(moved, out.roll(head_dim // 2, -1))


@pytest.mark.parametrize("batch", [2, 3, 4])
@pytest.mark.parametrize("hidden", [320, 1088, 2048])
def test_streaming_decode_of_a_few_sequences_gives_each_the_bits_it_gets_alone(device, batch, hidden):
    """Up to four sequences every sum is made in the same order, the squares of the norms among them: contexts of one tile are in
    one part, whatever the batch."""
    config = tiny_config(hidden=hidden, q_heads=8, kv_heads=4, head_dim=64, intermediate=1024, vocab=1000, layers=6)
    weights = synth_weights(config, seed=21, norm_std=0.1, device=device)
    together, alone = (make_kernel(config, weights, device, max_tokens=n, max_positions=12) for n in (batch, 1))
    states = [new_kv_state(config, n, 12, device) for n in (batch, *[1] * batch)]
    ids = synth_ids(batch * 12, config.vocab, seed=21).view(batch, 12).to(device)
    for position in range(12):
        positions = torch.full((batch, 1), position, dtype=torch.int64, device=device)
        step = ids[:, position:position + 1].contiguous()
        logits = together.decode(step, positions, *states[0])
        for row in range(batch):
            assert torch.equal(logits[row:row + 1], alone.decode(step[row:row + 1].contiguous(), positions[:1], *states[1 + row])), f"{row} at {position}"
    together.check()
    alone.check()

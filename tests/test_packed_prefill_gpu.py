"""Packed BF16 prefill steps (any number of rows of several prompts in one forward) at the sizes
where they can go wrong: query tiles and 128-position key tiles that are partly filled, prompts
around the window and around the 256 rows from which the linears run on CTA pairs, slots whose rings
hold an earlier, longer prompt. A row's result depends on its position and the keys it sees only, so
every cut of a prompt has to leave the same bytes; against the CPU oracle the bar is the one of
test_prefill_bf16_gpu.py.
"""
import pytest
import torch

import helpers
from helpers import rms_relative_error
from oracle import carat_semantics as cs
from test_prefill_bf16_gpu import build, prompts

pytestmark = pytest.mark.gpu

# Two and four query heads a KV head of 256, eight of 512.
CONFIG = cs.ModelConfig(256, 512, 2048, 256, 1024, 1e-6,
                        [cs.LayerConfig("sliding", 4, 2, 256, 1e4, False),
                         cs.LayerConfig("sliding", 4, 1, 256, 1e4, False),
                         cs.LayerConfig("global", 8, 1, 512, 1e6, True)])


def state(config, device, slot, length):
    rows = []
    for index in range(len(config.layers)):
        capacity = config.capacity(index)
        for cache in (device.key_cache(index, capacity), device.value_cache(index, capacity)):
            rows.append(cache[slot][:, :min(length, capacity)].contiguous().view(torch.int16))
    rows.append(device.target_hidden_slots()[slot].view(torch.int16))
    return rows


@pytest.mark.parametrize("length", [1, 16, 63, 129, 256, 257, 321, 640, 1000])
def test_every_cut_of_a_prompt_leaves_the_same_bytes(cuda_device, length):
    text = prompts(CONFIG, [length], seed=length)[0]
    other = prompts(CONFIG, [1000, 300], seed=5)
    _, device = build(CONFIG, 4)
    first = device.prefill_slot(0, text, chunk_tokens=1024)
    wanted = state(CONFIG, device, 0, length)
    # In pieces of 37 behind a longer prompt that used the slot before.
    device.prefill_slot(1, other[0], chunk_tokens=1024)
    assert device.prefill_slot(1, text, chunk_tokens=37) == first
    # Between two other prompts in one step, then in pieces of 130 beside one.
    device.prefill_slots_chunks([2, 3], [other[1], text], 1000)
    cuts = [1, 3]
    if length > 130:
        device.reset_slot(2)
        device.reset_slot(0)
        got = None
        while got is None:
            got = device.prefill_slots_chunks([0, 2], [text, other[0]], 130)[0]
        assert got == first
        cuts.append(0)
    for slot in cuts:
        for have, want in zip(state(CONFIG, device, slot, length), wanted):
            assert torch.equal(have, want), (length, slot)


def test_long_steps_match_the_oracle(cuda_device):
    lengths = [300, 517, 90]
    texts = prompts(CONFIG, lengths, seed=11)
    oracle, device = build(CONFIG, 3)
    wanted = [oracle.prefill_slot_fp8(slot, text, chunk=8) for slot, text in enumerate(texts)]
    got = device.prefill_slots_chunks([0, 1, 2], texts, 1024)    # 907 rows in one step
    assert sum(a != b for a, b in zip(got, wanted)) <= 1          # near-ties only
    for index in range(len(CONFIG.layers)):
        capacity = CONFIG.capacity(index)
        keys, values = device.key_cache(index, capacity), device.value_cache(index, capacity)
        for slot in range(3):
            assert rms_relative_error(keys[slot], oracle.keys[index][slot]) < 2e-2
            assert rms_relative_error(values[slot], oracle.values[index][slot]) < 2e-2
            assert helpers.cosine(keys[slot], oracle.keys[index][slot]) > 0.999


@pytest.mark.parametrize("context", [1024, 1000])
def test_rows_behind_the_last_token_do_not_count(cuda_device, context):
    """Cache rows that a prompt has not reached hold what was there before, and where the context is
    not whole key tiles the last tile reaches into the next head's and slot's rows: none of it may
    show, not even as 0 times an infinity."""
    config = cs.ModelConfig(CONFIG.hidden, CONFIG.intermediate, CONFIG.vocab, CONFIG.window, context,
                            CONFIG.eps, CONFIG.layers)
    lengths = [1, 130, 700, context]
    texts = prompts(config, lengths, seed=21)
    wanted = None
    for fill in (0.0, float("nan"), float("inf")):
        _, device = build(config, len(texts) + 1)
        for index, layer in enumerate(config.layers):
            rows = torch.full((len(texts) + 1, layer.kv_heads, config.capacity(index),
                               layer.head_dim), fill, dtype=torch.bfloat16)
            device.write_cache(0, index, rows)
            device.write_cache(1, index, rows)
        slots = list(range(len(texts)))
        tokens = device.prefill_slots_chunks(slots, texts, context)
        got = [state(config, device, slot, length) for slot, length in zip(slots, lengths)]
        if wanted is None:
            wanted = tokens, got
            continue
        assert tokens == wanted[0]
        for have, want in zip(got, wanted[1]):
            assert all(torch.equal(a, b) for a, b in zip(have, want))


def test_row_tiles_with_a_cut_tail_leave_the_same_bytes(cuda_device):
    """gate_up of 152 feature tiles (a round of 148 SMs and a last one cut along K), o in K pieces:
    together with the row tiles of more than 256 rows, every cut leaves the same bytes."""
    config = cs.ModelConfig(512, 9728, 2048, 256, 1024, 1e-6,
                            [cs.LayerConfig("sliding", 4, 2, 256, 1e4, False),
                             cs.LayerConfig("global", 8, 1, 512, 1e6, True)])
    length = 700
    text, other = prompts(config, [length, 900], seed=29)
    oracle, device = build(config, 5)
    first = device.prefill_slot(0, text, chunk_tokens=1024)       # three row tiles
    wanted = state(config, device, 0, length)
    assert device.prefill_slot(1, text, chunk_tokens=300) == first
    assert device.prefill_slot(2, text, chunk_tokens=67) == first
    assert device.prefill_slots_chunks([4, 3], [other, text], 1024)[1] == first   # 1,600 rows
    for slot in (1, 2, 3):
        for have, want in zip(state(config, device, slot, length), wanted):
            assert torch.equal(have, want), slot
    oracle.prefill_slot_fp8(0, text, chunk=8)
    for index in range(len(config.layers)):
        capacity = config.capacity(index)
        assert rms_relative_error(device.key_cache(index, capacity)[0], oracle.keys[index][0]) < 2e-2
        assert rms_relative_error(device.value_cache(index, capacity)[0],
                                  oracle.values[index][0]) < 2e-2


def test_a_feed_forward_width_without_small_divisors(cuda_device):
    """16 x 1,031 columns: the GeGLU row kernel of a step of many rows takes unequal parts."""
    config = cs.ModelConfig(256, 16 * 1031, 2048, 256, 512, 1e-6,
                            [cs.LayerConfig("sliding", 4, 2, 256, 1e4, False),
                             cs.LayerConfig("global", 8, 1, 512, 1e6, True)])
    text = prompts(config, [400], seed=31)[0]
    oracle, device = build(config, 2)
    first = device.prefill_slot(0, text, chunk_tokens=512)        # 400 rows: three parts
    assert device.prefill_slot(1, text, chunk_tokens=100) == first    # two
    for have, want in zip(state(config, device, 1, 400), state(config, device, 0, 400)):
        assert torch.equal(have, want)
    oracle.prefill_slot_fp8(0, text, chunk=8)
    for index in range(len(config.layers)):
        capacity = config.capacity(index)
        assert rms_relative_error(device.value_cache(index, capacity)[0],
                                  oracle.values[index][0]) < 2e-2

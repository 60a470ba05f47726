"""The eight-token prefill steps (the path of models whose query heads per KV head do not divide 128,
and of runners whose device had no room for the packed steps' buffers): head dimensions 256 and 512 on
the tensor-core attention kernels, rings read in place before the first wrap and wave by wave past it.
The bars are the ones of test_prefill_bf16_gpu.py."""
import pytest
import torch

import carat_b200
from helpers import cosine, rms_relative_error, runner_config
from oracle import carat_semantics as cs
from test_packed_prefill_gpu import state
from test_prefill_bf16_gpu import build, compare_state, prompts

pytestmark = pytest.mark.gpu

# Three query heads a KV head of 256, six of 512: neither divides the packed kernel's 128 rows.
CONFIG = cs.ModelConfig(256, 512, 2048, 256, 1024, 1e-6,
                        [cs.LayerConfig("sliding", 6, 2, 256, 1e4, False),
                         cs.LayerConfig("sliding", 3, 1, 256, 1e4, False),
                         cs.LayerConfig("global", 6, 1, 512, 1e6, True)])


def test_prompts_match_the_oracle(cuda_device):
    lengths = [64, 37, 300, 530]                   # the last two past the window of 256
    texts = prompts(CONFIG, lengths, seed=3)
    oracle, device = build(CONFIG, len(texts))
    wanted = [oracle.prefill_slot_fp8(slot, text, chunk=8) for slot, text in enumerate(texts)]
    got = [None] * len(texts)
    active = list(range(len(texts)))
    while active:
        results = device.prefill_slots_chunks(active, [texts[s] for s in active], 48)
        for slot, result in zip(list(active), results):
            if result is not None:
                got[slot] = result
                active.remove(slot)
    assert [device.slot_position(slot) for slot in range(4)] == lengths
    compare_state(CONFIG, oracle, device, range(4))
    table = device.target_hidden_slots()
    for slot in range(4):
        assert cosine(table[slot], oracle.target_hidden[slot]) > 0.999
    assert sum(a != b for a, b in zip(got, wanted)) <= 1          # near-ties only


@pytest.mark.parametrize("length", [9, 100, 256, 640])
def test_cuts_of_a_prompt(cuda_device, length):
    """Up to the first wrap every cut leaves the same bytes. Past it a row's sums begin with the rows of
    its own piece, and where pieces begin depends on the cut and on the prompts beside this one: fp32
    sums in another order, rounded to bf16, through three layers (the bars of the comparison with the
    oracle)."""
    text = prompts(CONFIG, [length], seed=length)[0]
    other = prompts(CONFIG, [300], seed=5)[0]
    _, device = build(CONFIG, 3)
    tokens = [device.prefill_slot(0, text, chunk_tokens=1024)]
    wanted = state(CONFIG, device, 0, length)
    tokens.append(device.prefill_slot(1, text, chunk_tokens=37))
    device.reset_slot(0)
    tokens.append(device.prefill_slots_chunks([2, 0], [text, other], 1000)[0])
    whole = length <= CONFIG.window
    assert not whole or len(set(tokens)) == 1
    for slot in (1, 2):
        *caches, hidden = zip(state(CONFIG, device, slot, length), wanted)
        for have, want in caches:
            if whole:
                assert torch.equal(have, want), (length, slot)
            assert rms_relative_error(have.view(torch.bfloat16), want.view(torch.bfloat16)) < 2e-2
        if whole:
            assert torch.equal(*hidden)
        assert cosine(hidden[0].view(torch.bfloat16), hidden[1].view(torch.bfloat16)) > 0.999


def test_a_device_without_room_for_the_packed_buffers(cuda_device):
    """The packed steps' staging alone takes 0.5 GB here. With less than that left the runner works in
    eight-token steps and holds on to nothing; with room again it packs."""
    slots = 24
    config = cs.ModelConfig(256, 512, 2048, 1024, 1280, 1e-6,
                            [cs.LayerConfig("sliding", 16, 16, 256, 1e4, False),
                             cs.LayerConfig("global", 8, 1, 512, 1e6, True)])
    weights = cs.golden_tiny_weights(config)
    arena = carat_b200.DeviceWeightArena.from_host(weights)
    fp8 = carat_b200.Fp8WeightArena.quantize(arena)
    device = carat_b200.Gemma4BatchModelRunner(runner_config(config), arena, slots,
                                               config.max_context, fp8)
    texts = prompts(config, [1100, 40, 333], seed=13)
    torch.cuda.empty_cache()
    left = 256 << 20
    filler = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")
    free = torch.cuda.mem_get_info()[0]
    device.set_bf16_weights()
    held = free - torch.cuda.mem_get_info()[0]
    assert held < 64 << 20
    walked = device.prefill_slots_chunks([0, 1, 2], texts, 2048)
    del filler
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    device.set_bf16_weights()
    assert free - torch.cuda.mem_get_info()[0] > 512 << 20
    packed = device.prefill_slots_chunks([3, 4, 5], texts, 2048)
    assert sum(a != b for a, b in zip(walked, packed)) <= 1       # near-ties only
    for index, layer in enumerate(config.layers):
        capacity = config.capacity(index)
        for cache in (device.key_cache(index, capacity), device.value_cache(index, capacity)):
            for slot, text in enumerate(texts):
                rows = slice(0, min(len(text), capacity))
                assert rms_relative_error(cache[3 + slot][:, rows], cache[slot][:, rows]) < 2e-2
    table = device.target_hidden_slots()
    for slot in range(3):
        assert cosine(table[3 + slot], table[slot]) > 0.999

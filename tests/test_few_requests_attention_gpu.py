"""Global attention of a few requests, whose contexts of more than 512 rows are cut into chunks of 256 to
512 while each chunk has an SM to itself, against the CUDA-core kernels (which do not cut by that rule), through the
runner against the oracle, and under stream capture. The bar against the CUDA-core kernels is the one
of the tensor-core attention's other comparisons: 2e-2 of the largest output."""
import subprocess
import sys

import pytest
import torch

import carat_b200
from carat_b200.capi import check
from conftest import ROOT
from helpers import relative_error, rms_relative_error
from test_runner_tc_parity_gpu import GLOBAL, build_seeded_pair, small_real_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth", [1, 5])
@pytest.mark.parametrize("contexts", [[513], [600, 40], [1024], [3000], [1200, 1, 2047, 700, 700],
                                      [900] * 24])
def test_cut_contexts_match_the_cuda_core_kernels(cuda_device, contexts, depth):
    library = carat_b200.library()
    generator = torch.Generator(device="cuda").manual_seed(len(contexts) + depth)
    requests, heads, kv_heads, dim = len(contexts), 32, 4, 512
    longest = max(contexts)
    capacity = (longest + depth + 127) // 128 * 128

    def normal(*shape):
        return (torch.randn(*shape, device="cuda", generator=generator) * 0.3).to(torch.bfloat16)

    queries = normal(requests, heads, depth, dim)
    keys, values = normal(requests, kv_heads, capacity, dim), normal(requests, kv_heads, capacity, dim)
    twins = len(contexts) > 4 and contexts[3] == contexts[4]
    if twins:
        for tensor in (queries, keys, values):       # equal requests have to come out equal
            tensor[4] = tensor[3]
    positions = torch.tensor(contexts, dtype=torch.int32, device="cuda")
    stride = 16 + (longest + depth + 127) // 128 * 128
    scores = torch.empty(requests * heads * depth * stride, dtype=torch.bfloat16, device="cuda")
    results = []
    for entry in (library.carat_b200_verify_attention, library.carat_b200_verify_attention_check):
        out = torch.full((requests * depth, heads * dim), float("nan"), dtype=torch.bfloat16,
                         device="cuda")
        check(entry(queries.data_ptr(), keys.data_ptr(), values.data_ptr(), None, None,
                    positions.data_ptr(), out.data_ptr(), scores.data_ptr(), stride, requests,
                    depth, heads, kv_heads, dim, capacity, 0, longest, None))
        torch.cuda.synchronize()
        results.append(out)
    got, want = results
    assert relative_error(got, want) < 2e-2
    if twins:
        rows = got.view(requests, depth, -1).view(torch.int16)
        assert torch.equal(rows[3], rows[4])


@pytest.mark.parametrize("slots", [[1], [0], [0, 1]])
def test_a_verify_step_of_few_slots_matches_the_oracle(cuda_device, slots):
    """One global layer; the slots stand at 700 and 2,100 of 2,304 positions. The bar is the one of
    the full batch's one-layer step, which is not cut."""
    config = small_real_config([GLOBAL])
    oracle, device = build_seeded_pair(config)
    depth = 5
    generator = torch.Generator().manual_seed(17)
    proposals = torch.randint(3, config.vocab, (len(slots), depth), generator=generator).tolist()
    firsts = [row[0] for row in proposals]
    caps = [depth] * len(slots)
    _, _, trace = oracle.verify_greedy_proposals(proposals, firsts, slots, caps, assume_match=True,
                                                 trace=True)
    result = device.verify_greedy_proposals(proposals, firsts, slots, caps,
                                            carat_b200.VERIFY_ASSUME_MATCH)
    assert result.accepted_tokens == caps
    hidden = device.last_final_hidden(len(slots) * depth)
    assert rms_relative_error(hidden, trace.final_hidden) < 0.02


CAPTURED = """
import torch
import carat_b200
from carat_b200.capi import check
library = carat_b200.library()
depth, heads, kv_heads, dim, capacity = 5, 32, 4, 512, 1024

def call(requests, length):
    generator = torch.Generator(device="cuda").manual_seed(requests)
    def normal(*shape):
        return (torch.randn(*shape, device="cuda", generator=generator) * 0.3).to(torch.bfloat16)
    queries = normal(requests, heads, depth, dim)
    keys, values = normal(requests, kv_heads, capacity, dim), normal(requests, kv_heads, capacity, dim)
    positions = torch.full((requests,), length, dtype=torch.int32, device="cuda")
    stride = 16 + capacity
    scores = torch.empty(requests * heads * depth * stride, dtype=torch.bfloat16, device="cuda")
    out = torch.empty(requests * depth, heads * dim, dtype=torch.bfloat16, device="cuda")
    def run():
        check(library.carat_b200_verify_attention(
            queries.data_ptr(), keys.data_ptr(), values.data_ptr(), None, None, positions.data_ptr(),
            out.data_ptr(), scores.data_ptr(), stride, requests, depth, heads, kv_heads, dim, capacity,
            0, length, torch.cuda.current_stream().cuda_stream))
        return out
    return run

call(24, 900)()                    # a full batch first: not cut, so no partial sums are kept
few = call(2, 900)
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    captured = few()
captured.zero_()
graph.replay()
torch.cuda.synchronize()
got = captured.clone()
want = few()
torch.cuda.synchronize()
assert (got.float() - want.float()).abs().max() < 2e-2 * want.float().abs().max()
print("captured")
"""


def test_a_call_of_few_requests_can_be_captured(cuda_device):
    """A stream under capture cannot get scratch for the cut: the call takes the uncut form then. In a
    process of its own, whose scratch no other test has grown."""
    done = subprocess.run([sys.executable, "-c", CAPTURED], cwd=ROOT, capture_output=True, text=True,
                          timeout=300)
    assert done.returncode == 0 and "captured" in done.stdout, done.stderr[-2000:]

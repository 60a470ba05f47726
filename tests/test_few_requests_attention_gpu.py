"""Global attention of a few requests, whose contexts are cut into chunks of 256 rows and more until
every SM has one, against the CUDA-core kernels (which do not cut by that rule). The bar is the one of
the tensor-core attention's other comparisons: 2e-2 of the largest output."""
import pytest
import torch

import carat_b200
from carat_b200.capi import check
from helpers import relative_error

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

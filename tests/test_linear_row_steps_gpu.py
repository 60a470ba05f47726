"""The linear at the edges of its row variants (UMMA N in steps of 32, each with its own ring depth)
and of its finishing kernels (vector and column form, K pieces and tail columns), against fp32. A
call of few rows and one of many take every sum in the same order, so their common rows are
bit-equal; the norm-wise bar against fp32 is twice the bf16 rounding of the output (2^-9).
"""
import pytest
import torch

import carat_b200
from carat_b200.capi import check
from helpers import rms_relative_error

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 32, 33, 65, 96, 97, 128, 129, 160, 192, 193, 224, 225, 256])
@pytest.mark.parametrize("k,n", [(2048, 5376), (1024, 20480), (1040, 5320), (512, 1000)])
def test_rows_at_the_edges_of_the_variants(cuda_device, rows, k, n):
    library = carat_b200.library()
    generator = torch.Generator(device="cuda").manual_seed(k + n)
    x, x_scale = carat_b200.quantize_tensor_to_fp8(
        torch.randn(256, k, device="cuda", generator=generator).to(torch.bfloat16))
    w, w_scale = carat_b200.quantize_tensor_to_fp8(
        (torch.randn(n, k, device="cuda", generator=generator) * 0.02).to(torch.bfloat16))

    def linear(count):
        out = torch.full((count, n), float("nan"), dtype=torch.bfloat16, device="cuda")
        size = library.carat_b200_fp8_linear_workspace_bytes(count, k, n)
        workspace = torch.empty(max(size, 16), dtype=torch.uint8, device="cuda")
        check(library.carat_b200_fp8_linear(
            x.data_ptr(), x_scale.data_ptr(), w.data_ptr(), w_scale.data_ptr(), out.data_ptr(),
            count, k, n, workspace.data_ptr(), size, None))
        torch.cuda.synchronize()
        return out

    got = linear(rows)
    want = ((x[:rows].view(torch.float8_e4m3fn).float() @ w.view(torch.float8_e4m3fn).float().t())
            * (x_scale * w_scale))
    assert rms_relative_error(got, want) < 4e-3
    assert torch.equal(got[:1].view(torch.int16), linear(1).view(torch.int16))


@pytest.mark.parametrize("rows", [1, 96, 97, 160, 161, 224, 225])
@pytest.mark.parametrize("k,n", [(2048, 5376), (1024, 20480), (520, 1000)])
def test_bf16_rows_at_the_edges_of_the_variants(cuda_device, rows, k, n):
    library = carat_b200.library()
    generator = torch.Generator(device="cuda").manual_seed(k + n)
    x = torch.randn(256, k, device="cuda", generator=generator).to(torch.bfloat16)
    w = (torch.randn(n, k, device="cuda", generator=generator) * 0.02).to(torch.bfloat16)

    def linear(count):
        out = torch.full((count, n), float("nan"), dtype=torch.bfloat16, device="cuda")
        size = library.carat_b200_bf16_linear_workspace_bytes(count, k, n)
        workspace = torch.empty(max(size, 16), dtype=torch.uint8, device="cuda")
        check(library.carat_b200_bf16_linear(x.data_ptr(), w.data_ptr(), out.data_ptr(), count, k, n,
                                             workspace.data_ptr(), size, None))
        torch.cuda.synchronize()
        return out

    got = linear(rows)
    assert rms_relative_error(got, x[:rows].float() @ w.float().t()) < 4e-3
    assert torch.equal(got[:1].view(torch.int16), linear(1).view(torch.int16))

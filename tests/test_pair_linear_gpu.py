"""The linear's CTA-pair kernel (calls of many rows) against fp32 and against the single-CTA kernel.

Both kernels take every sum in the same order (the K pieces and the K-cut tail depend on the widths
only), so a row's result may not depend on how many rows its call has: bit-equal, not close.
Against fp32 the bar is the bf16 rounding of the output, 2^-9 relative to a value, plus the
accumulation order; 4e-3 norm-wise is twice that rounding's worst case.
"""
import ctypes

import pytest
import torch

import carat_b200
from carat_b200.capi import check
from helpers import rms_relative_error

pytestmark = pytest.mark.gpu

# (rows of the wide call, K, N): edges of the row tile, odd 128-feature tile counts, a K-cut tail,
# a last feature tile that is half empty, K that is not a whole number of blocks.
SHAPES = [(161, 4096, 16384), (193, 4096, 16384), (193, 5376, 43008), (224, 4112, 19200), (256, 5376, 18944 + 128),
          (255, 8192, 9472 + 64)]


@pytest.mark.parametrize("wide", [False, True], ids=["e4m3", "bf16"])
@pytest.mark.parametrize("rows,k,n", SHAPES)
def test_rows_do_not_depend_on_the_call_they_are_in(cuda_device, wide, rows, k, n):
    library = carat_b200.library()
    generator = torch.Generator(device="cuda").manual_seed(rows + n)
    x = torch.randn(rows, k, device="cuda", generator=generator).to(torch.bfloat16)
    w = (torch.randn(n, k, device="cuda", generator=generator) * 0.02).to(torch.bfloat16)
    if not wide:
        x, x_scale = carat_b200.quantize_tensor_to_fp8(x)
        w, w_scale = carat_b200.quantize_tensor_to_fp8(w)

    def linear(count):
        out = torch.full((count, n), float("nan"), dtype=torch.bfloat16, device="cuda")
        size = (library.carat_b200_bf16_linear_workspace_bytes if wide
                else library.carat_b200_fp8_linear_workspace_bytes)(count, k, n)
        workspace = torch.empty(max(size, 16), dtype=torch.uint8, device="cuda")
        if wide:
            check(library.carat_b200_bf16_linear(x.data_ptr(), w.data_ptr(), out.data_ptr(), count,
                                                 k, n, workspace.data_ptr(), size, None))
        else:
            check(library.carat_b200_fp8_linear(
                x.data_ptr(), x_scale.data_ptr(), w.data_ptr(), w_scale.data_ptr(),
                out.data_ptr(), count, k, n, workspace.data_ptr(), size, None))
        torch.cuda.synchronize()
        return out

    many = linear(rows)
    few = linear(100)
    assert torch.equal(many[:100].view(torch.int16), few.view(torch.int16))
    if wide:
        want = x.float() @ w.float().t()
    else:
        want = ((x.view(torch.float8_e4m3fn).float() @ w.view(torch.float8_e4m3fn).float().t())
                * (x_scale * w_scale))
    assert rms_relative_error(many, want) < 4e-3


@pytest.mark.parametrize("wide", [False, True], ids=["e4m3", "bf16"])
@pytest.mark.parametrize("rows", [97, 120, 193, 224, 256])
def test_argmax_on_pairs(cuda_device, wide, rows):
    """The LM head's epilogue: against fp32 logits, and token for token against the single-CTA kernel
    (calls of 96 rows and fewer; both take every sum in the same order). The features that win are
    planted twice or more: in one warp, in the two CTAs of a pair, in one half tile beside the end, and
    in other tiles; the lowest index has to win each time."""
    library = carat_b200.library()
    k, n = 4096, 160064                  # 32 (e4m3) and 64 blocks of K; the last tile holds 64 features
    generator = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, k, device="cuda", generator=generator).to(torch.bfloat16)
    w = (torch.randn(n, k, device="cuda", generator=generator) * 0.02).to(torch.bfloat16)
    twins = [(5, 9), (70, 200), (130, 250), (300, 300 + 256), (1000, n - 1), (n - 64, n - 2),
             (40000, 41000, 90000)]
    for row, group in enumerate(twins):
        w[list(group)] = x[row] * 0.5    # far ahead of the other logits of this row
    if not wide:
        x, x_scale = carat_b200.quantize_tensor_to_fp8(x)
        w, w_scale = carat_b200.quantize_tensor_to_fp8(w)

    def tokens(first, count):
        out = torch.empty(count, dtype=torch.int32, device="cuda")
        keys = torch.empty(count, dtype=torch.int64, device="cuda")
        part = x[first:first + count]
        if wide:
            check(library.carat_b200_bf16_linear_argmax(part.data_ptr(), w.data_ptr(), out.data_ptr(),
                                                        keys.data_ptr(), count, k, n, None))
        else:
            check(library.carat_b200_fp8_linear_argmax(
                part.data_ptr(), x_scale.data_ptr(), w.data_ptr(), w_scale.data_ptr(),
                out.data_ptr(), keys.data_ptr(), count, k, n, None))
        torch.cuda.synchronize()
        return out.cpu()

    got = tokens(0, rows)
    assert got[:len(twins)].tolist() == [min(group) for group in twins]
    alone = torch.cat([tokens(first, min(96, rows - first)) for first in range(0, rows, 96)])
    assert torch.equal(got, alone)
    if wide:
        logits = x.float() @ w.float().t()
    else:
        logits = ((x.view(torch.float8_e4m3fn).float() @ w.view(torch.float8_e4m3fn).float().t())
                  * (x_scale * w_scale))
    chosen = logits.gather(1, got.cuda().long()[:, None])[:, 0]
    top = logits.max(1).values
    assert bool((top - chosen <= top.abs() * 2.0 ** -7).all())      # one bf16 rounding of a logit


def test_kernels_that_follow_a_pair_on_its_sms(cuda_device):
    """Pair launches of one and several tiles a pair, each followed at once by a kernel whose barriers
    lie where the pair's lay: an arrival left over from the pair would count there. Every round leaves
    the same bytes and no wait runs out."""
    library = carat_b200.library()
    generator = torch.Generator(device="cuda").manual_seed(3)
    calls = []
    for rows, k, n in ((256, 2048, 18944), (24, 1024, 5376), (200, 4096, 37888), (5, 512, 18944)):
        x = torch.randn(rows, k, device="cuda", generator=generator).to(torch.bfloat16)
        w = (torch.randn(n, k, device="cuda", generator=generator) * 0.02).to(torch.bfloat16)
        out = torch.empty(rows, n, dtype=torch.bfloat16, device="cuda")
        size = library.carat_b200_bf16_linear_workspace_bytes(rows, k, n)
        calls.append((x, w, out, rows, k, n, torch.empty(max(size, 16), dtype=torch.uint8,
                                                         device="cuda"), size))

    def round_of_calls():
        for x, w, out, rows, k, n, workspace, size in calls:
            check(library.carat_b200_bf16_linear(x.data_ptr(), w.data_ptr(), out.data_ptr(), rows,
                                                 k, n, workspace.data_ptr(), size, None))

    round_of_calls()
    torch.cuda.synchronize()
    first = [call[2].clone() for call in calls]
    for _ in range(10):
        for _ in range(50):
            round_of_calls()
        torch.cuda.synchronize()
        for call, want in zip(calls, first):
            assert torch.equal(call[2].view(torch.int16), want.view(torch.int16))
    code = ctypes.c_int(0)
    check(library.carat_b200_device_error(ctypes.byref(code)))
    assert code.value == 0

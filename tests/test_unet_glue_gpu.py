"""The kernels between the U-Net's convolutions against torch.

Copies are exact; the pooled mean is a sum of eight BF16 values in FP32 rounded
once, so it differs from the FP64 mean by the final rounding (2^-9 relative) and
FP32 sums (8 x 2^-24 of the largest term)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(1, 2, 2, 2, 8), (1, 4, 2, 6, 16), (2, 6, 10, 4, 24), (3, 8, 8, 8, 48), (1, 34, 18, 26, 32)]


def _stream():
    return torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("shape", SHAPES)
def test_pool(shape):
    from langevinfts_b200.capi import check, lib
    B, D, H, W, C = shape
    torch.manual_seed(1)
    x = torch.randn(shape, device="cuda").to(torch.bfloat16)
    x[0, 0, 0, 0, 0] = float("inf")
    y = torch.full([B, D // 2, H // 2, W // 2, C], 7.0, device="cuda", dtype=torch.bfloat16)
    check(lib().lfts_unet_pool_bf16(_stream(), x.data_ptr(), y.data_ptr(), B, D, H, W, C))
    blocks = x.double().reshape(B, D // 2, 2, H // 2, 2, W // 2, 2, C)
    want, big = blocks.mean((2, 4, 6)), blocks.abs().amax((2, 4, 6))
    assert torch.isinf(y[0, 0, 0, 0, 0])
    y[0, 0, 0, 0, 0] = want[0, 0, 0, 0, 0] = big[0, 0, 0, 0, 0] = 0.0
    assert torch.all((y.double() - want).abs() <= want.abs() * 2.0 ** -8 + big * 2.0 ** -21)


@pytest.mark.parametrize("ca,cb", [(8, 8), (96, 48), (48, 32), (16, 40)])
@pytest.mark.parametrize("shape", SHAPES)
def test_upsample_and_concatenate(shape, ca, cb):
    from langevinfts_b200.capi import check, lib
    B, D, H, W, _ = shape
    torch.manual_seed(2)
    a = torch.randn([B, D // 2, H // 2, W // 2, ca], device="cuda").to(torch.bfloat16)
    b = torch.randn([B, D, H, W, cb], device="cuda").to(torch.bfloat16)
    y = torch.empty([B, D, H, W, ca + cb], device="cuda", dtype=torch.bfloat16)
    check(lib().lfts_unet_upcat_bf16(_stream(), a.data_ptr(), b.data_ptr(), y.data_ptr(), B, D, H, W, ca, cb))
    up = a.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)
    assert torch.equal(y, torch.cat([up, b], -1))


@pytest.mark.parametrize("cin,cpad", [(1, 8), (2, 16), (3, 16), (16, 16), (17, 32)])
@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (2, 3, 5, 7), (1, 16, 20, 12)])
def test_pack_input(shape, cin, cpad):
    from langevinfts_b200.capi import check, lib
    B, D, H, W = shape
    torch.manual_seed(3)
    x = torch.randn([B, cin, D, H, W], device="cuda")
    y = torch.full([B, D, H, W, cpad], 7.0, device="cuda", dtype=torch.bfloat16)
    check(lib().lfts_unet_pack_input(_stream(), x.data_ptr(), y.data_ptr(), B, cin, D, H, W, cpad))
    want = torch.nn.functional.pad(x.permute(0, 2, 3, 4, 1).to(torch.bfloat16), (0, cpad - cin))
    assert torch.equal(y, want)


def test_refusals():
    from langevinfts_b200.capi import lib
    x = torch.zeros(4096, device="cuda", dtype=torch.bfloat16)
    p = x.data_ptr()
    assert lib().lfts_unet_pool_bf16(_stream(), p, p, 1, 3, 2, 2, 8) != 0
    assert lib().lfts_unet_pool_bf16(_stream(), p, p, 1, 2, 2, 2, 12) != 0
    assert lib().lfts_unet_upcat_bf16(_stream(), p, p + 2, p, 1, 2, 2, 2, 8, 8) != 0
    assert lib().lfts_unet_pack_input(_stream(), p, p, 1, 9, 2, 2, 2, 8) != 0

"""Saturating E4M3 cast at the edges of its blocks of rows, on dense and strided tensors."""
import pytest
import torch

import dtb200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [1, 15, 16, 127, 128, 129, 400])
@pytest.mark.parametrize("strided", [False, True])
def test_cast_equals_the_torch_cast_bit_for_bit(S, strided):
    g = torch.Generator(device="cuda").manual_seed(S)
    shape = (2, S, 3, 128) if strided else (2, 3, S, 128)
    x = (torch.randn(shape, generator=g, device="cuda") * 200).to(torch.bfloat16)
    if strided:
        x = x.transpose(1, 2)
    got = dtb200.quantize_e4m3(x, mult=1.25)
    want = (x.float() * 1.25).clamp(-448, 448).to(torch.float8_e4m3fn)
    assert got.shape == x.shape and got.is_contiguous()
    assert torch.equal(got.view(torch.uint8), want.contiguous().view(torch.uint8))

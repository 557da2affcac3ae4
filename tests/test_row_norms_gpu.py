"""Per-head row-norm maxima at the sizes where the split into blocks and rows in flight can go wrong."""
import pytest
import torch

from dtb200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [1, 7, 8, 63, 65, 255, 256, 257, 1031])
def test_row_norm_maxima_over_block_edges(S):
    g = torch.Generator(device="cuda").manual_seed(S)
    q = torch.randn(2, 6, S, 128, generator=g, device="cuda").to(torch.bfloat16)
    k = torch.randn(2, S, 3, 128, generator=g, device="cuda").to(torch.bfloat16).transpose(1, 2)
    # the largest row of each head sits at another place: last row, first row, anywhere
    q[1, 0, S - 1] *= 4
    q[0, 1, 0] *= 4
    k[1, 2, S - 1] *= 4
    qn, kn = ops.row_norm_maxima(q, k)
    mult = 128 ** -0.5 * 1.44269504
    want_q = q.double().norm(dim=-1).amax(dim=(0, 2)) * mult
    want_k = k.double().norm(dim=-1).amax(dim=(0, 2))
    # 128 squares summed in f32 in a tree of depth 7, a square root and a product: below 16 roundings of 2^-24
    assert ((qn.double() - want_q).abs() / want_q).max().item() <= 16 * 2.0 ** -24
    assert ((kn.double() - want_k).abs() / want_k).max().item() <= 16 * 2.0 ** -24


def test_row_norm_maxima_of_zeros_are_zero():
    z = torch.zeros(1, 2, 300, 128, dtype=torch.bfloat16, device="cuda")
    qn, kn = ops.row_norm_maxima(z, z)
    assert qn.abs().max().item() == 0.0 and kn.abs().max().item() == 0.0

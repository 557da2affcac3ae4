"""128-row blocks, whose softmax groups take alternate key tiles of one query tile, beside 256-row blocks.

Few heads: the launch is cut into 128-row blocks.  Many heads: 256-row blocks.  Key tile counts of 1, 2, 3, ... are the
edges of the alternation.  Tolerance: bf16 probabilities and outputs, as in the other parity tests."""
import pytest
import torch

import dtb200
from oracle import attn_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(B, H, Sq, Skv, seed, gain=1.0):
    g = torch.Generator().manual_seed(seed)
    q, k, v = (torch.randn(B, H, s, 128, generator=g) for s in (Sq, Skv, Skv))
    q = q * torch.rsqrt(q.pow(2).mean(-1, keepdim=True)) * gain
    k = k * torch.rsqrt(k.pow(2).mean(-1, keepdim=True))
    return tuple(t.to(torch.bfloat16) for t in (q, k, v))


def _check(out, ref, peak=None):
    # bf16 rounds to half a unit of 2^-7: at most 2^-8 of a probability, at most 2^-8 of an output.  With near one-hot
    # rows neither averages out, and an output is as large as its value row: 2^-7 of the largest value in all.
    dtb200.check_device_status(DEV)
    err = (out.float().cpu() - ref).abs()
    assert err.max().item() <= (2e-2 if peak is None else 2.0 ** -7 * peak) and err.mean().item() <= 2e-3, (err.max().item(), err.mean().item())


@pytest.mark.parametrize("H", [2, 148])
@pytest.mark.parametrize("Sq,Skv", [(1, 1), (77, 128), (128, 129), (129, 384), (300, 500), (384, 640), (333, 1111)])
@pytest.mark.parametrize("gain", [1.0, 12.0])
def test_ragged_ends(H, Sq, Skv, gain):
    q, k, v = _inputs(1, H, Sq, Skv, seed=Sq + Skv, gain=gain)
    if gain > 1.0:     # peaks in later key tiles: the two groups' offsets move, and differ
        k[:, :, Skv // 2] *= 3
    out = dtb200.attention(q.to(DEV), k.to(DEV), v.to(DEV), zero_padded_rows=False)
    _check(out, O.attention_fp32(q, k, v), peak=v.abs().max().item() if gain > 1.0 else None)


@pytest.mark.parametrize("H", [2, 148])
@pytest.mark.parametrize("pad", [40, 170, 256, 300])
def test_padded_second_tile_is_zero(H, pad):
    S = 512
    q, k, v = _inputs(2, H, S, S, seed=pad)
    kv_len = torch.tensor([S, S - pad], dtype=torch.int32)
    out = torch.full((2, H, S, 128), float("nan"), dtype=torch.bfloat16, device=DEV)
    dtb200.attention(q.to(DEV), k.to(DEV), v.to(DEV), kv_len=kv_len.to(DEV), out=out)
    _check(out, O.attention_fp32(q, k, v, kv_len=kv_len))
    assert out[1, :, S - pad:].abs().max().item() == 0.0


@pytest.mark.parametrize("H", [2, 148])
def test_ring_steps_fixed_offset_and_fp8(H):
    Sq, Skv = 333, 450
    q, k, v = _inputs(1, H, Sq, 2 * Skv, seed=5)
    qd, kd, vd = (t.to(DEV) for t in (q, k, v))
    ref = O.attention_fp32(q, k, v, kv_len=[2 * Skv - 30])
    mk = dtb200.fixed_m_operands(qd, kd, gate=213.0)
    for kw in ({}, {"use_fixed_m": True, "mk": mk}):
        state = dtb200.ResidualState(1, H, Sq, qd.device)
        for i in range(2):
            part = slice(i * Skv, (i + 1) * Skv)
            dtb200.residual_attention_(state, qd, kd[:, :, part], vd[:, :, part], kv_len=[2 * Skv - 30], kv_offset=i * Skv, **kw)
        _check(dtb200.finalize_residual(state), ref)
    q8, k8 = dtb200.quantize_e4m3(qd, mult=128 ** -0.5 * 1.44269504), dtb200.quantize_e4m3(kd)
    ref8 = O.attention_fp32(q8.float().cpu(), k8.float().cpu(), v, scale=1 / 1.44269504, kv_len=[2 * Skv - 30])
    out = dtb200.attention(qd, kd, vd, qk_fp8=True, kv_len=[2 * Skv - 30], zero_padded_rows=False)
    _check(out, ref8)


@pytest.mark.parametrize("H,Sq,Skv", [(24, 333, 6000), (24, 100, 6000), (2, 100, 6000)])
def test_short_queries_against_many_keys(H, Sq, Skv):
    """Sizes on both sides of the choice between 128-row blocks and a last wave cut into pieces."""
    q, k, v = _inputs(1, H, Sq, Skv, seed=9)
    out = dtb200.attention(q.to(DEV), k.to(DEV), v.to(DEV), kv_len=[Skv - 100], zero_padded_rows=False)
    _check(out, O.attention_fp32(q, k, v, kv_len=[Skv - 100], zero_padded_rows=False))

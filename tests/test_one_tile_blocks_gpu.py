"""128-row blocks, whose softmax groups take alternate key tiles of one query tile, beside 256-row blocks.

The choice follows from the shape, so every test asserts which form runs.  Key tile counts of 1, 2, 3, ... are the edges of
the alternation; 128-row blocks reach them through the valid length, since a key tensor that short goes to 256-row blocks.
Tolerance: bf16 probabilities and outputs, as in the other parity tests."""
import ctypes

import pytest
import torch

import dtb200
from dtb200 import _lib, ops
from oracle import attn_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _block_rows(q, k):
    """Query rows of a CTA of the launch that these tensors lead to: none of them is cut into pieces."""
    assert "plain launch" in dtb200.describe_launch(*q.shape[:3], k.shape[2])
    p = ops._fill_params(q, k, k, None, None, None, None, 0, 0, None)
    return _lib.load().dtb_attn_block_rows(ctypes.byref(p), None, 0)


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


def _peaked(k, at):
    """A key that outweighs the others in a later key tile: the two groups' offsets move, and differ."""
    k[:, :, at] *= 3
    return k


@pytest.mark.parametrize("Sq", [1, 77, 128, 129, 300])
@pytest.mark.parametrize("keys", [1, 128, 129, 384, 500, 640, 750, 1111, 2048])     # 1, 1, 2, 3, 4, 5, 6, 9 and 16 key tiles
@pytest.mark.parametrize("gain", [1.0, 12.0])
def test_ragged_ends_128_row_blocks(Sq, keys, gain):
    q, k, v = _inputs(1, 2, Sq, 2048, seed=Sq + keys, gain=gain)
    if gain > 1.0:
        k = _peaked(k, keys // 2)
    qd, kd, vd = (t.to(DEV) for t in (q, k, v))
    assert _block_rows(qd, kd) == 128
    out = dtb200.attention(qd, kd, vd, kv_len=[keys], zero_padded_rows=False)
    _check(out, O.attention_fp32(q, k[:, :, :keys], v[:, :, :keys]), peak=v.abs().max().item() if gain > 1.0 else None)


@pytest.mark.parametrize("H", [2, 148])
@pytest.mark.parametrize("Sq,Skv", [(1, 1), (77, 128), (128, 129), (129, 384), (300, 500), (384, 640), (333, 1111)])
@pytest.mark.parametrize("gain", [1.0, 12.0])
def test_ragged_ends(H, Sq, Skv, gain):
    q, k, v = _inputs(1, H, Sq, Skv, seed=Sq + Skv, gain=gain)
    if gain > 1.0:
        k = _peaked(k, Skv // 2)
    qd, kd, vd = (t.to(DEV) for t in (q, k, v))
    assert _block_rows(qd, kd) == (128 if H == 2 and Skv in (500, 1111) else 256)
    out = dtb200.attention(qd, kd, vd, zero_padded_rows=False)
    _check(out, O.attention_fp32(q, k, v), peak=v.abs().max().item() if gain > 1.0 else None)


@pytest.mark.parametrize("H", [2, 148])
@pytest.mark.parametrize("pad", [40, 170, 256, 300])
def test_padded_second_tile_is_zero(H, pad):
    S = 512
    q, k, v = _inputs(2, H, S, S, seed=pad)
    kv_len = torch.tensor([S, S - pad], dtype=torch.int32)
    out = torch.full((2, H, S, 128), float("nan"), dtype=torch.bfloat16, device=DEV)
    assert _block_rows(q.to(DEV), k.to(DEV)) == (128 if H == 2 else 256)
    dtb200.attention(q.to(DEV), k.to(DEV), v.to(DEV), kv_len=kv_len.to(DEV), out=out)
    _check(out, O.attention_fp32(q, k, v, kv_len=kv_len))
    assert out[1, :, S - pad:].abs().max().item() == 0.0


@pytest.mark.parametrize("H", [2, 148])
@pytest.mark.parametrize("last", [1, 129, 300, 420])      # keys of the second step: 1, 2, 3 and 4 tiles on top of a state
def test_ring_steps_fixed_offset_and_fp8(H, last):
    Sq, Skv = 333, 450
    q, k, v = _inputs(1, H, Sq, 2 * Skv, seed=5)
    kv_len = [Skv + last]
    qd, kd, vd = (t.to(DEV) for t in (q, k, v))
    assert _block_rows(qd, kd[:, :, :Skv]) == _block_rows(qd, kd) == (128 if H == 2 else 256)
    ref = O.attention_fp32(q, k, v, kv_len=kv_len, zero_padded_rows=False)
    mk = dtb200.fixed_m_operands(qd, kd, gate=213.0)
    for kw in ({}, {"use_fixed_m": True, "mk": mk}):
        state = dtb200.ResidualState(1, H, Sq, qd.device)
        for i in range(2):
            part = slice(i * Skv, (i + 1) * Skv)
            dtb200.residual_attention_(state, qd, kd[:, :, part], vd[:, :, part], kv_len=kv_len, kv_offset=i * Skv, **kw)
        _check(dtb200.finalize_residual(state), ref)
    q8, k8 = dtb200.quantize_e4m3(qd, mult=128 ** -0.5 * 1.44269504), dtb200.quantize_e4m3(kd)
    ref8 = O.attention_fp32(q8.float().cpu(), k8.float().cpu(), v, scale=1 / 1.44269504, kv_len=kv_len, zero_padded_rows=False)
    out = dtb200.attention(qd, kd, vd, qk_fp8=True, kv_len=kv_len, zero_padded_rows=False)
    _check(out, ref8)


@pytest.mark.parametrize("H,Sq,Skv,form", [(24, 333, 6000, "cut into"), (24, 100, 6000, "cut into"), (2, 100, 6000, "cut into"),
                                           (48, 333, 4000, "128 rows"), (48, 600, 4000, "per query block")])
def test_short_queries_against_many_keys(H, Sq, Skv, form):
    """Sizes on each side of the choice between 128-row blocks, 256-row blocks and a last wave cut into pieces."""
    assert form in dtb200.describe_launch(1, H, Sq, Skv)
    q, k, v = _inputs(1, H, Sq, Skv, seed=9)
    out = dtb200.attention(q.to(DEV), k.to(DEV), v.to(DEV), kv_len=[Skv - 100], zero_padded_rows=False)
    _check(out, O.attention_fp32(q, k, v, kv_len=[Skv - 100], zero_padded_rows=False))


def test_128_row_blocks_over_131_key_tiles():
    q, k, v = _inputs(1, 48, 333, 16731, seed=11)
    assert _block_rows(q.to(DEV), k.to(DEV)) == 128
    out = dtb200.attention(q.to(DEV), k.to(DEV), v.to(DEV), kv_len=[16700], zero_padded_rows=False)
    _check(out, O.attention_fp32(q, k, v, kv_len=[16700], zero_padded_rows=False))


@pytest.mark.parametrize("words", [4, 8, 12])
@pytest.mark.parametrize("Sq", [77, 300])
@pytest.mark.parametrize("second", ["online", "bounded", "e4m3"])
def test_a_running_state_may_start_at_any_multiple_of_16_bytes(words, Sq, second):
    """128-row blocks read it 32 bytes at a time where it allows that and 16 where not: the same state either way."""
    q, k, v = (t.to(DEV) for t in _inputs(1, 2, Sq, 2048, seed=Sq))
    mk = dtb200.fixed_m_operands(q, k) if second == "bounded" else None
    states = []
    for at in (0, words):
        state = dtb200.ResidualState(1, 2, Sq, q.device)
        state.o = torch.full((2 * Sq * 128 + 16,), float("nan"), device=DEV)[at:at + 2 * Sq * 128].view(1, 2, Sq, 128)
        assert state.o.data_ptr() % 64 == 4 * at and _block_rows(q, k[:, :, :1024]) == 128
        # after an online step the bounded one finds a state relative to another offset than its own
        dtb200.residual_attention_(state, q, k[:, :, :1024], v[:, :, :1024])
        dtb200.residual_attention_(state, q, k[:, :, 1024:], v[:, :, 1024:], kv_offset=1024, use_fixed_m=second == "bounded", mk=mk,
                                   qk_fp8=second == "e4m3")
        states.append(state)
    dtb200.check_device_status(DEV)
    for a, b in zip(*((s.o, s.m, s.l) for s in states)):
        assert torch.equal(a, b)
    _check(dtb200.finalize_residual(states[1]), O.attention_fp32(*(t.cpu() for t in (q, k, v))), peak=v.abs().max().item() if second == "e4m3" else None)

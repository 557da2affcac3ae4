"""NaN and infinity in the inputs come out as they do from float32 attention, whichever kernel and key tile meets them."""
import ctypes

import pytest
import torch

import dtb200
from dtb200 import _lib, ops

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")
SQ, SKV = 300, 1280                      # ten key tiles
KERNELS = [(2, 128), (60, 256)]          # heads, rows of a CTA that this many heads lead to


def _inputs(H, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    q, k, v = (torch.randn(1, H, s, 128, generator=g, device=DEV) for s in (SQ, SKV, SKV))
    q, k = (t * torch.rsqrt(t.pow(2).mean(-1, keepdim=True)) for t in (q, k))
    return tuple(t.to(torch.bfloat16) for t in (q, k, v))


def _reference(q, k, v):
    return torch.softmax(q.float() @ k.float().transpose(-1, -2) * 128 ** -0.5, -1) @ v.float()


def _run(kind, q, k, v, rows):
    p = ops._fill_params(q, k, v, None, None, None, None, 0, 1, None)
    assert _lib.load().dtb_attn_block_rows(ctypes.byref(p), None, 0) == rows
    if kind == "plain":
        out = dtb200.attention(q, k, v, num_splits=1)
    else:                                # a second ring step meets the keys; the first one holds a copy of the first key tile
        state = dtb200.ResidualState(1, q.shape[1], SQ, DEV)
        dtb200.residual_attention_(state, q, k[:, :, :128], v[:, :, :128])
        dtb200.residual_attention_(state, q, k, v, kv_offset=128)
        out = state.o / state.l[..., None]
    dtb200.check_device_status(DEV)
    return out.float()


def _merged(kind, q, k, v, kv_len=None):
    """Calls whose results are merged from partial states by a kernel of their own."""
    if kind == "ring":
        state = dtb200.ResidualState(*q.shape[:3], DEV)
        dtb200.residual_attention_(state, q, k, v, kv_len=kv_len)
        out = dtb200.finalize_residual(state, kv_len=kv_len)
    elif kind == "splits":
        out = dtb200.attention(q, k, v, kv_len=kv_len, num_splits=3)
    else:
        assert "cut into" in dtb200.describe_launch(*q.shape[:3], k.shape[2])
        out = dtb200.attention(q, k, v, kv_len=kv_len)
    dtb200.check_device_status(DEV)
    return out.float()


def _check(out, ref):
    assert torch.equal(out.isnan(), ref.isnan())
    # bf16 probabilities and outputs, as in the other parity tests
    assert (out - ref).nan_to_num(0.0).abs().max().item() <= 2e-2


@pytest.mark.parametrize("H,rows", KERNELS)
@pytest.mark.parametrize("kind", ["plain", "ring"])
@pytest.mark.parametrize("what", ["nan", "inf", "value"])
@pytest.mark.parametrize("key", [5, 130, 270, 1100, 1279])     # key tiles 0, 1, 2, 8 and 9
def test_not_a_number_reaches_the_output(H, rows, kind, what, key):
    q, k, v = _inputs(H, key)
    if what == "nan":                    # every row of head 0 is NaN, no other head is
        k[0, 0, key] = float("nan")
    elif what == "value":                # one column of head 0 is NaN
        v[0, 0, key, 7] = float("nan")
    else:                                # logits of +inf for rows with q[0] > 0 (NaN), of -inf for the others (weight 0)
        k[0, 0, key, 0] = 3e38
        q[0, 0, :, 0] = torch.where(torch.arange(SQ, device=DEV) % 3 == 0, 2.0, -2.0).to(torch.bfloat16)
    ref = _reference(q, k, v) if kind == "plain" else _reference(q, torch.cat([k[:, :, :128], k], 2), torch.cat([v[:, :, :128], v], 2))
    assert ref.isnan().any()
    _check(_run(kind, q, k, v, rows), ref)


@pytest.mark.parametrize("H,rows", KERNELS)
@pytest.mark.parametrize("kind", ["plain", "ring"])
@pytest.mark.parametrize("tiles", [(1,), (1, 2), (2, 3), (1, 3, 5, 7, 9), (9,)])
@pytest.mark.parametrize("every", [1, 3])
def test_key_tiles_whose_logits_are_all_minus_infinity_weigh_nothing(H, rows, kind, tiles, every):
    q, k, v = _inputs(H, tiles[-1])
    q[..., 0] = torch.where(torch.arange(SQ, device=DEV) % every == 0, 2.0, 0.0).to(torch.bfloat16)   # the other rows see them
    for t in tiles:
        k[:, :, 128 * t:128 * t + 128, 0] = -3e38
    ref = _reference(q, k, v) if kind == "plain" else _reference(q, torch.cat([k[:, :, :128], k], 2), torch.cat([v[:, :, :128], v], 2))
    assert not ref.isnan().any()
    _check(_run(kind, q, k, v, rows), ref)


@pytest.mark.parametrize("kind,H,S,first", [("ring", 1, 300, 0), ("ring", 2, 1280, 0), ("ring", 60, 1280, 1), ("splits", 1, 1280, 0),
                                            ("splits", 1, 1280, 1), ("pieces", 1, 4608, 0), ("pieces", 1, 4608, 1), ("pieces", 12, 4608, 1)])
def test_partial_states_that_start_with_minus_infinity_keep_their_other_keys(kind, H, S, first):
    """Every other key tile, from ``first`` on, is all -inf for two rows of three; some states begin with such a tile."""
    g = torch.Generator(device=DEV).manual_seed(S + first)
    q, k, v = (torch.randn(1, H, S, 128, generator=g, device=DEV) for _ in range(3))
    q, k = (t * torch.rsqrt(t.pow(2).mean(-1, keepdim=True)) for t in (q, k))
    q[..., 0] = torch.where(torch.arange(S, device=DEV) % 3 == 0, 0.0, 2.0)
    k[..., 0] = torch.where(torch.arange(S, device=DEV) // 128 % 2 == first, -3e38, 0.5)
    q, k, v = (t.to(torch.bfloat16) for t in (q, k, v))
    out = _merged(kind, q, k, v)
    for h in range(H):
        _check(out[:, h], _reference(q[:, h], k[:, h], v[:, h]))


@pytest.mark.parametrize("kind,S", [("ring", 500), ("splits", 1280), ("pieces", 4608)])
@pytest.mark.parametrize("tile", [0, 1, 2, 3])
def test_not_a_number_passes_through_a_merge(kind, S, tile):
    g = torch.Generator(device=DEV).manual_seed(tile)
    q, k, v = (torch.randn(1, 1, S, 128, generator=g, device=DEV).to(torch.bfloat16) for _ in range(3))
    k[0, 0, 128 * tile + 9, 0] = 3e38                       # +inf or -inf, by the sign of q
    q[..., 0] = torch.where(torch.arange(S, device=DEV) % 3 == 0, 2.0, -2.0).to(torch.bfloat16)
    ref = _reference(q, k, v)
    assert ref.isnan().any() and not ref.isnan().all()
    out = _merged(kind, q, k, v)
    assert torch.equal(out.isnan(), ref.isnan())


@pytest.mark.parametrize("kind,S", [("ring", 500), ("splits", 1280), ("pieces", 4608)])
def test_a_merge_zeroes_padded_queries_whatever_they_hold(kind, S):
    g = torch.Generator(device=DEV).manual_seed(S)
    q, k, v = (torch.randn(1, 1, S, 128, generator=g, device=DEV).to(torch.bfloat16) for _ in range(3))
    q[:, :, S - 70:] = float("nan")
    out = _merged(kind, q, k, v, kv_len=[S - 70])
    assert out[:, :, S - 70:].abs().max().item() == 0.0 and not out.isnan().any()

"""Launches of a few dozen query blocks: pieces of 256-row blocks or whole 128-row blocks.

The lines asserted are those of the rule beside ``kSecondPieceTiles`` in ``attn_api.cu``, a comparison of two modelled times in which
the one of the pieces has a surcharge where there are more of them than SMs; 1 x 2 x 3328 and 1 x 2 x 6144 stay in pieces by it
although they are the slower form there.  On the GPU the calls that it gives to 128-row blocks agree with float32 attention, and
with key splits on 256-row blocks, in the layouts that an entry point takes."""
import pytest
import torch

import dtb200

POLICY = [  # B, heads, rows, 128-row blocks?
    (1, 1, 3072, False), (1, 2, 3072, False), (1, 1, 9216, False), (1, 2, 6144, False), (1, 3, 16896, False), (1, 12, 4608, False),
    (1, 2, 3328, False),
    (1, 3, 2560, True), (1, 3, 2816, True), (1, 3, 3072, True), (1, 3, 4608, True), (1, 4, 3072, True), (2, 2, 3072, True), (1, 3, 5200, True), (1, 2, 9216, True),
]


@pytest.mark.parametrize("B,H,S,rows128", POLICY)
def test_more_pieces_than_sms_give_way_to_128_row_blocks(B, H, S, rows128):
    line = dtb200.describe_launch(B, H, S, sms=148)
    assert ("per 128 rows" in line) == rows128 and ("pieces" in line) != rows128, line


@pytest.mark.gpu
@pytest.mark.parametrize("B,H,Hkv,Sq,Skv,kv_len,layout", [
    (1, 3, 3, 3072, 3072, None, "bhsd"),
    (1, 3, 3, 3001, 3001, [2870], "bshd"),
    (2, 2, 1, 3072, 3072, [3072, 2817], "bhsd"),
    (1, 4, 2, 2999, 3137, [3130], "bshd"),
])
def test_moved_calls_agree_with_both_references(B, H, Hkv, Sq, Skv, kv_len, layout):
    g = torch.Generator(device="cuda").manual_seed(Sq)

    def make(heads, rows):
        shape = (B, heads, rows, 128) if layout == "bhsd" else (B, rows, heads, 128)
        x = torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16)
        return x if layout == "bhsd" else x.transpose(1, 2)

    q, k, v = make(H, Sq), make(Hkv, Skv), make(Hkv, Skv)
    assert "per 128 rows" in dtb200.describe_launch(B, H, Sq, Skv)
    lens = None if kv_len is None else torch.tensor(kv_len, dtype=torch.int32, device="cuda")
    got = dtb200.attention(q, k, v, kv_len=lens, zero_padded_rows=False)
    split = dtb200.attention(q, k, v, kv_len=lens, zero_padded_rows=False, num_splits=2)
    dtb200.check_device_status()
    for b in range(B):
        n = Skv if kv_len is None else kv_len[b]
        kk, vv = (t[b, :, :n].float().repeat_interleave(H // Hkv, 0) for t in (k, v))
        want = torch.softmax(q[b].float() @ kk.transpose(1, 2) * 128 ** -0.5, -1) @ vv
        for out in (got, split):     # bf16 probabilities and results: half a unit of 2^-8 of values up to 1, and a margin
            err = (out[b].float() - want).abs()
            assert err.max().item() <= 2e-2 and err.mean().item() <= 2e-3

"""Decode attention with more blocks than the GPU holds at a time: the blocks take the rows in the order
of their lengths, which changes no result.  Compared bit for bit with the same rows in calls of 30 (few
enough for the plain order, the same kernel otherwise) and with f32 attention; up to 128 rows are
ordered, more are not."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

NQ, NKV, HD, SEQ = 16, 8, 64, 160


def positions_of(kind, batch, gen):
    mixed = torch.randint(0, SEQ, (batch,), generator=gen)
    if kind == "equal":
        return torch.full((batch,), SEQ - 1)
    if kind == "pairs":  # every length twice, in falling order
        return torch.arange(batch).flip(0) // 2 % SEQ
    return mixed


def inputs(batch, gen):
    q = torch.randn(batch, NQ, HD, generator=gen).to(torch.bfloat16).cuda()
    k = torch.randn(batch, NKV, SEQ, HD, generator=gen).to(torch.bfloat16).cuda()
    v = torch.randn(batch, NKV, SEQ, HD, generator=gen).to(torch.bfloat16).cuda()
    return q, k, v


@pytest.mark.parametrize("batch", [38, 64, 127, 128, 129])
@pytest.mark.parametrize("kind", ["equal", "pairs", "mixed"])
def test_row_order_changes_nothing(batch, kind):
    from linnet_b200 import glue

    gen = torch.Generator().manual_seed(batch)
    q, k, v = inputs(batch, gen)
    positions = positions_of(kind, batch, gen).cuda()
    got = glue.decode_attention(q, k, v, positions, splits=1)
    for r0 in range(0, batch, 30):
        part = slice(r0, min(batch, r0 + 30))
        if part.stop - r0 < 20:
            part = slice(batch - 30, batch)  # 20 rows or more: blocks of as many warps
        assert torch.equal(got[part], glue.decode_attention(q[part], k[part], v[part], positions[part], splits=1))
    mask = (torch.arange(SEQ, device="cuda")[None, :] <= positions[:, None])[:, None, None, :]
    want = torch.nn.functional.scaled_dot_product_attention(
        q.float()[:, :, None], k.float(), v.float(), attn_mask=mask, enable_gqa=True).reshape(batch, NQ * HD)
    torch.testing.assert_close(got.float(), want, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("batch", [64, 128])
@pytest.mark.parametrize("bad", [SEQ, -1, 1 << 40, -(1 << 40)])
def test_a_bad_position_among_many_rows(batch, bad):
    """Its row means nothing and is reported; the others are as without it."""
    from linnet_b200 import glue

    gen = torch.Generator().manual_seed(batch)
    q, k, v = inputs(batch, gen)
    positions = positions_of("mixed", batch, gen).cuda()
    want = glue.decode_attention(q, k, v, positions, splits=1)
    glue.decoder_status()
    spoiled, row = positions.clone(), batch // 2
    spoiled[row] = bad
    got = glue.decode_attention(q, k, v, spoiled, splits=1)
    torch.cuda.synchronize()
    with pytest.raises(ValueError, match=f"batch row {row}"):
        glue.decoder_status()
    glue.decoder_status()
    others = [i for i in range(batch) if i != row]
    assert torch.equal(got[others], want[others])


def test_fused_attention_of_many_rows():
    """Rotary embedding and cache write in the same launch: every row writes its own key."""
    from linnet_b200 import glue

    batch = 100
    gen = torch.Generator().manual_seed(3)
    _, k, v = inputs(batch, gen)
    qkv = torch.randn(batch, (NQ + 2 * NKV) * HD, generator=gen).to(torch.bfloat16).cuda()
    positions = positions_of("mixed", batch, gen).cuda()
    table = glue.rope_table(SEQ, HD, 1e4, torch.device("cuda", 0))
    k1, v1, k2, v2 = k.clone(), v.clone(), k.clone(), v.clone()
    got = glue.rope_attention(qkv, positions, table, k1, v1, NQ, NKV, splits=1)
    for r0 in range(0, batch, 25):
        part = slice(r0, r0 + 25)
        assert torch.equal(got[part], glue.rope_attention(qkv[part], positions[part], table, k2[part], v2[part], NQ, NKV,
                                                          splits=1))
    assert torch.equal(k1, k2) and torch.equal(v1, v2)

"""Decode attention of several lanes with eight key heads and more: two CTAs per SM, a row's bits whatever the number of rows (B200 only)."""

import pytest
import torch

from tests import test_gpu_namizen as single

pytestmark = pytest.mark.gpu


# tiles of 64 keys: chunks around one and several, more query heads per key head than one tile of eight, heads that pad, wide heads, more than 32 key heads
@pytest.mark.parametrize("shape", [(32, 8, 128, 128, 700, 1024), (16, 8, 96, 80, 64, 512), (80, 8, 128, 112, 65, 256), (8, 8, 48, 64, 300, 512), (16, 16, 128, 128, 130, 512),
                                   (8, 8, 200, 256, 130, 512), (40, 40, 128, 128, 100, 256)])
def test_several_lanes(native_lib, shape):
    single.test_decode_attention(native_lib, shape, False)


# six rows on long rings: two parts of the keys to a CTA (eight key heads, also padded ones), splits by the rows (nine and twenty heads, values of 64, wide heads)
@pytest.mark.parametrize("shape", [(32, 8, 128, 128, 3000, 4096), (16, 8, 96, 80, 2049, 4096), (80, 8, 128, 112, 2100, 4096), (18, 9, 128, 128, 2500, 4096),
                                   (20, 20, 64, 128, 2200, 4096), (20, 20, 64, 64, 2200, 4096), (9, 9, 256, 200, 2100, 4096)])
def test_several_lanes_on_long_rings(native_lib, shape):
    single.test_decode_attention(native_lib, shape, False)


@pytest.mark.parametrize("H,G,dim", [(32, 8, 128), (32, 8, 64), (16, 16, 128)])
def test_a_rows_bits_do_not_depend_on_the_others(native_lib, H, G, dim):
    lanes, ring, positions = 8, 1024, [1000, 5, 517, 63, 64, 1023, 200, 900]
    gen = torch.Generator(device="cuda").manual_seed(H + dim)
    draw = lambda *s: torch.randn(s, device="cuda", generator=gen).to(torch.bfloat16)  # noqa: E731
    q, k, v = draw(lanes, H, dim), draw(lanes, ring, G, dim), draw(lanes, ring, G, dim)
    pos, lane, sink = torch.tensor(positions, dtype=torch.int32, device="cuda"), torch.arange(lanes, dtype=torch.int32, device="cuda"), torch.zeros(H, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    results = []
    for rows in (2, 3, 8):
        out = torch.zeros((rows, H * dim), dtype=torch.bfloat16, device="cuda")
        a = single.attention_args(native_lib, q[:rows], k, v, sink, dim**-0.5, out, H, G, dim, dim, status)
        a.row_pos, a.row_lane, a.row_active = pos.data_ptr(), lane.data_ptr(), None
        a.rows, a.decode, a.chunk, a.ring, a.capacity, a.lanes = rows, 1, ring, ring, ring, lanes
        native_lib.chunk_attention(a, False)
        results.append(out)
    assert int(status) == 0
    assert torch.equal(results[0], results[2][:2]) and torch.equal(results[1], results[2][:3])


# three, four and eight key heads (also with two blocks of query heads in a fragment), sixteen of 64, head sizes of every kernel: a part of the keys per CTA
# and two, parts of unequal length and without a key
@pytest.mark.parametrize("H,G,dim", [(12, 3, 128), (16, 4, 64), (32, 8, 128), (80, 8, 128), (32, 8, 64), (16, 16, 64), (32, 8, 256)])
def test_a_rows_bits_deep_in_a_ring(native_lib, H, G, dim):
    lanes, ring, positions = 8, 8192, [8000, 63, 5017, 8191, 64, 3000, 511, 1]
    gen = torch.Generator(device="cuda").manual_seed(G + dim)
    draw = lambda *s: torch.randn(s, device="cuda", generator=gen).to(torch.bfloat16)  # noqa: E731
    q, k, v = draw(lanes, H, dim), draw(lanes, ring, G, dim), draw(lanes, ring, G, dim)
    pos, lane, sink = torch.tensor(positions, dtype=torch.int32, device="cuda"), torch.arange(lanes, dtype=torch.int32, device="cuda"), torch.zeros(H, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")

    def rows_of(rows):
        out = torch.full((rows, H * dim), float("nan"), dtype=torch.bfloat16, device="cuda")
        a = single.attention_args(native_lib, q[:rows], k, v, sink, dim**-0.5, out, H, G, dim, dim, status)
        a.row_pos, a.row_lane, a.row_active = pos.data_ptr(), lane.data_ptr(), None
        a.rows, a.decode, a.chunk, a.ring, a.capacity, a.lanes = rows, 1, ring, ring, ring, lanes
        native_lib.chunk_attention(a, False)
        return out

    all_rows = rows_of(8)
    for rows in range(2, 8):
        assert torch.equal(rows_of(rows), all_rows[:rows]), rows
    assert int(status) == 0
    for r in (0, 1, 5):
        n = positions[r] + 1
        keys, values = (t[r, :n].double().repeat_interleave(H // G, 1) for t in (k, v))
        score = torch.einsum("hd,jhd->hj", q[r].double(), keys) * dim**-0.5
        weight = torch.exp(score - score.amax(1, keepdim=True).clamp(min=0))
        weight = weight / (weight.sum(1, keepdim=True) + torch.exp(-score.amax(1, keepdim=True).clamp(min=0)))  # the sink's score is 0
        want = torch.einsum("hj,jhd->hd", weight, values).flatten()
        # products and sums in fp32 (weights as two bf16 pieces), one rounding to bf16: 2^-9 / sqrt(3) = 1.1e-3 in the 2-norm
        assert float((all_rows[r].double() - want).norm() / want.norm()) < 2e-3, r

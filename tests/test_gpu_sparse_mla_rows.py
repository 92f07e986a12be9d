"""Sparse attention of many query rows at the flagship's head shape (64 heads, latent 512, rotary 64): the tensor-core kernel."""

import pytest
import torch

pytestmark = pytest.mark.gpu

H, L, RD = 64, 512, 64
W = L + RD


def _case(counts, top_k, cap, seed, spread=1.0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rows = len(counts)
    q = (torch.randn(rows, H, W, device="cuda", generator=gen) * spread).to(torch.bfloat16)
    cache = torch.randn(2, 2, cap, W, device="cuda", generator=gen).to(torch.bfloat16)  # two lanes, two layers
    sel = torch.stack([torch.randperm(cap, device="cuda", generator=gen)[:top_k] for _ in range(rows)]).to(torch.int32)
    sel = sel.sort(dim=1).values.contiguous()
    cnt = torch.tensor([[c, c] for c in counts], dtype=torch.int32, device="cuda")
    lane = torch.ones(rows, dtype=torch.int32, device="cuda")
    return q, cache, sel, cnt, lane


def _run(native, q, cache, sel, cnt, lane, top_k, scale):
    rows = q.shape[0]
    out = torch.full((rows, H, L), float("nan"), dtype=torch.bfloat16, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    native.sparse_mla_rows(q, cache, sel, cnt, lane, rows, H, L, RD, 1, 2, cache.shape[2], top_k, scale, out, status)
    torch.cuda.synchronize()
    return out, int(status)


def _exact(q, cache, sel, counts, scale):
    out = torch.zeros(q.shape[0], H, L, dtype=torch.float64, device="cuda")
    for r, c in enumerate(counts):
        if c:
            k = cache[1, 1, sel[r, :c].long()].double()
            out[r] = torch.softmax(q[r].double() @ k.T * scale, dim=1) @ k[:, :L]
    return out


# edges of the sixteen-key steps and the 128-key blocks, more rows than CTAs, empty rows; ``spread``: how sharp the softmax is (wide scores
# make the running maximum move after the first block)
@pytest.mark.parametrize("counts,spread", [
    ([1], 0.3), ([0, 1, 15, 16, 17, 127, 128, 129], 0.3), ([255, 256, 257, 2048, 0, 2047], 0.3), ([640, 1900], 4.0),
    ([(37 * i) % 300 for i in range(470)], 0.6),
])
def test_rows_against_64_bits(native_lib, counts, spread):
    top_k, cap = max(16, max(counts)), 4096
    q, cache, sel, cnt, lane = _case(counts, top_k, cap, seed=len(counts), spread=spread)
    scale = W**-0.5
    out, status = _run(native_lib, q, cache, sel, cnt, lane, top_k, scale)
    assert status == 0
    want = _exact(q, cache, sel, counts, scale)
    for r, c in enumerate(counts):
        if not c:
            assert not out[r].any()
            continue
        # the weights and the result are rounded to bf16 (2^-9 / sqrt(3) = 1.1e-3 each in the 2-norm); twice their sum
        err = float((out[r].double() - want[r]).norm() / want[r].norm())
        assert err < 4.5e-3, (r, c, err)


def test_growing_scores_follow_the_maximum_and_bad_rows_are_reported(native_lib):
    """Keys in rising order of their score: the reference of the exponents has to move in block after block."""
    count, cap = 1024, 2048
    q, cache, sel, cnt, lane = _case([count], count, cap, seed=5)
    q[0] = q[0, :1].abs()
    cache[1, 1] = cache[1, 1].abs() * torch.linspace(0.02, 1.0, cap, device="cuda")[:, None].to(torch.bfloat16)
    scale = 0.5  # scores from a few units to about 150
    out, status = _run(native_lib, q, cache, sel, cnt, lane, count, scale)
    assert status == 0
    want = _exact(q, cache, sel, [count], scale)
    assert float((out[0].double() - want[0]).norm() / want[0].norm()) < 4.5e-3
    bad = sel.clone()
    bad[0, 700] = cap + 3  # clamped and reported, as by the general kernel
    _, status = _run(native_lib, q, cache, bad, cnt, lane, count, scale)
    assert status == native_lib.STATUS_BAD_INDEX
    q[0, 3, 7] = float("inf")
    _, status = _run(native_lib, q, cache, sel, cnt, lane, count, scale)
    assert status & native_lib.STATUS_NONFINITE


@pytest.mark.parametrize("count,spread", [(200, 1.0), (2048, 0.3), (2048, 1.0), (2048, 4.0), (2048, 12.0)])
def test_rounding_the_weights_costs_what_it_must(native_lib, count, spread):
    """The error is that of weights rounded to bf16 beside the heaviest, which is 1, and of a rounded result; however sharp the softmax is."""
    rows, cap = 24, 4096
    q, cache, sel, cnt, lane = _case([count] * rows, count, cap, seed=3, spread=spread)
    scale = W**-0.5
    out, status = _run(native_lib, q, cache, sel, cnt, lane, count, scale)
    assert status == 0
    got, best, size = 0.0, 0.0, 0.0
    for r in range(rows):
        k = cache[1, 1, sel[r, :count].long()].double()
        score = q[r].double() @ k.T * scale
        weight = torch.exp(score - score.max(dim=1, keepdim=True).values)
        total = weight.sum(dim=1, keepdim=True)
        want = weight @ k[:, :L] / total
        rounded = (weight.to(torch.bfloat16).double() @ k[:, :L] / total).to(torch.bfloat16).double()
        got += float((out[r].double() - want).square().sum())
        best += float((rounded - want).square().sum())
        size += float(want.square().sum())
    # the maximum is that of the blocks so far: a few weights of early blocks are rounded beside a smaller one, by the same 2^-9 at most
    assert got**0.5 <= 1.06 * best**0.5, (got / size, best / size)

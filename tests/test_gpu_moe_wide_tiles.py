"""Tiles of more than 64 routes, whose results the decode warps help to store, have the bits of the same routes in tiles of up to 64 (B200 only)."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,N", [(16, 136), (128, 1024), (384, 1024), (1040, 264)])  # 1, 1, 3 and 9 steps; several items per CTA
def test_results_do_not_depend_on_the_tiles(native_lib, K, N):
    n = native_lib
    gen = torch.Generator(device="cuda").manual_seed(K)
    counts = [65, 128, 81, 96, 7, 112, 80, 64, 127] * 9
    P, el = sum(counts), len(counts)
    w = [(torch.randn(el, N, K, device="cuda", generator=gen) * 64).clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8) for _ in range(2)]
    s = [(torch.rand(el, -(-N // 128), -(-K // 128), device="cuda", generator=gen) + 0.5) * (K**-0.5 / 64) for _ in range(2)]
    x = torch.randn(P, K, device="cuda", generator=gen).bfloat16()
    perm = torch.randperm(P, device="cuda", generator=gen).int()
    weight = torch.rand(P, device="cuda", generator=gen) + 0.1
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    results = []
    for most in (128, 64):
        tiles, start = [], 0
        for e, c in enumerate(counts):
            tiles += [[r, min(r + most, start + c), e, 0] for r in range(start, start + c, most)]
            start += c
        listed, count = torch.tensor(tiles, dtype=torch.int32, device="cuda"), torch.tensor([len(tiles)], dtype=torch.int32, device="cuda")
        act, dw = (torch.full((P, N), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2))
        n.moe_grouped_fp8w(x, *w, *s, listed, count, 0, act, status=status)
        n.moe_grouped_fp8w(x, w[0], None, s[0], None, listed, count, 1, dw, perm=perm, route_weight=weight, status=status)
        results.append((act, dw))
    assert int(status) == 0
    assert all(not a.isnan().any() and torch.equal(a, b) for a, b in zip(*results))

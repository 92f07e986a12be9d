"""Route sums of many rows: eight columns a thread, the bits of the sums in route order."""

import pytest
import torch

pytestmark = pytest.mark.gpu


# one 16-byte piece, a ragged second block of columns, route counts off the step of four, columns that are no whole pieces, rows of a decode step
@pytest.mark.parametrize("rows,top_k,H", [(9, 1, 8), (11, 8, 2056), (300, 6, 264), (10, 5, 36), (8, 8, 64)])
@pytest.mark.parametrize("offset", [0, 1], ids=["aligned", "unaligned"])
def test_route_sums(native_lib, rows, top_k, H, offset):
    n = native_lib
    gen = torch.Generator().manual_seed(rows * top_k)
    E, base = 6, 2
    ids = torch.randint(0, E + 4, (rows, top_k), generator=gen).to(torch.int32)  # some of other GPUs, below and above
    flat = torch.full((offset + rows * top_k * H,), float("nan"), dtype=torch.bfloat16)
    dw = flat[offset:].view(rows * top_k, H)
    local = ((ids >= base) & (ids < base + E)).flatten()
    dw[local] = torch.randn(int(local.sum()), H, generator=gen).to(torch.bfloat16)  # the others are never read
    shared = torch.randn(rows, H, generator=gen)
    routed = torch.zeros(rows, H)
    for s in range(top_k):
        routed += torch.where(local.view(rows, top_k)[:, s, None], dw.view(rows, top_k, H)[:, s].float(), torch.zeros(()))
    bf = lambda t: t.to(torch.bfloat16).float()  # noqa: E731
    want = (bf(bf(routed) * 2.5) + bf(shared)).to(torch.bfloat16)
    dw_d = flat.cuda()[offset:].view(rows * top_k, H)
    out, partial = torch.zeros(rows, H, dtype=torch.bfloat16, device="cuda"), torch.zeros(rows, H, device="cuda")
    n.moe_combine(dw_d, ids.cuda(), shared.cuda(), rows, top_k, H, base, E, 2.5, False, out)
    n.moe_combine(dw_d, ids.cuda(), None, rows, top_k, H, base, E, 2.5, False, None, partial)
    torch.cuda.synchronize()
    assert torch.equal(out.cpu(), want) and torch.equal(partial.cpu(), routed)

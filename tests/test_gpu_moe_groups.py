"""Decode experts read once for the routes that chose them: the bits of the kernels with a CTA per route (B200 only)."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# routes that all differ, that all agree (more than eight to an expert), other GPUs' experts, an expert twice in a row; column blocks with a ragged end, K of
# fewer steps than warps and a multiple of 64 only
@pytest.mark.parametrize("rows,tk,E,ebase,el,H,I,same", [
    (4, 8, 64, 0, 64, 6144, 2048, False), (8, 8, 16, 0, 16, 1088, 1040, False), (5, 8, 4, 0, 4, 448, 2064, True), (8, 6, 32, 8, 16, 960, 4096, False),
])
def test_grouped_routes_have_the_bits_of_a_cta_per_route(native_lib, rows, tk, E, ebase, el, H, I, same):
    n = native_lib
    gen = torch.Generator(device=DEV).manual_seed(rows * tk + H)
    codes = lambda *s: torch.randint(0, 256, s, dtype=torch.uint8, device=DEV, generator=gen).bitwise_and_(0xBF)  # noqa: E731  (no NaN)
    blocks = lambda a, b: torch.rand((el, -(-a // 128), -(-b // 128)), device=DEV, generator=gen) * 0.1  # noqa: E731
    wg, wu, wd = codes(el, I, H), codes(el, I, H), codes(el, H, I)
    sg, su, sd = blocks(I, H), blocks(I, H), blocks(H, I)
    x = torch.randn((rows, H), device=DEV, generator=gen).to(torch.bfloat16)
    weight = torch.rand((rows, tk), device=DEV, generator=gen)
    if same:
        ids = torch.full((rows, tk), E - 1, device=DEV)
        ids[1, :3] = 0
    else:
        ids = torch.rand((rows, E), device=DEV, generator=gen).argsort(dim=1)[:, :tk].clone()
        ids[0, 1] = ids[0, 0]
    ids = ids.to(torch.int32).contiguous()
    P = rows * tk
    own = ((ids >= ebase) & (ids < ebase + el)).flatten()

    def run(routes):  # all of them in one launch, or one after another: a single route always has a CTA per tile
        act = torch.full((P, I), float("nan"), dtype=torch.bfloat16, device=DEV)
        dw = torch.full((P, H), float("nan"), dtype=torch.bfloat16, device=DEV)
        flat, w = ids.flatten(), weight.flatten()
        for p in routes:
            at = slice(0, P) if p is None else slice(p, p + 1)
            rows_in = x if p is None else x[p // tk : p // tk + 1]
            count = P if p is None else 1
            n.moe_gateup_fp8(rows_in, tk, flat[at].contiguous(), None, None, count, 1, wg, wu, sg, su, ebase, act[at])
            n.moe_down_fp8(act[at], w[at].contiguous(), flat[at].contiguous(), None, None, count, 1, wd, sd, ebase, dw[at])
        return act, dw

    together, alone = run([None]), run(range(P))
    for a, b in zip(together, alone):
        assert torch.equal(a[own], b[own]) and bool(a[~own].isnan().all())
        assert bool(a[own].isfinite().all())


def test_fewer_steps_than_warps(native_lib):
    """K of 64: one warp has a step, the others add zeros."""
    n = native_lib
    gen = torch.Generator(device=DEV).manual_seed(3)
    E, H, I, rows, tk = 8, 64, 8192, 8, 4
    wg, wu = (torch.randint(0, 256, (E, I, H), dtype=torch.uint8, device=DEV, generator=gen).bitwise_and_(0xBF) for _ in range(2))
    s = torch.rand((E, I // 128, 1), device=DEV, generator=gen) * 0.1
    x = torch.randn((rows, H), device=DEV, generator=gen).to(torch.bfloat16)
    ids = torch.rand((rows, E), device=DEV, generator=gen).argsort(dim=1)[:, :tk].to(torch.int32).contiguous()
    act = torch.zeros((rows * tk, I), dtype=torch.bfloat16, device=DEV)
    n.moe_gateup_fp8(x, tk, ids, None, None, rows * tk, 1, wg, wu, s, s, 0, act)
    full = s.repeat_interleave(128, 1)
    g, u = ((w.view(torch.float8_e4m3fn).float() * full).bfloat16().double() for w in (wg, wu))
    for p in range(rows * tk):
        e = int(ids.flatten()[p])
        z, v = x[p // tk].double() @ g[e].T, x[p // tk].double() @ u[e].T
        want = z * torch.sigmoid(z) * v
        # both factors are rounded to bf16 (2^-9 each, the gate's slope at most 1.1), and so is the result
        assert ((act[p].double() - want).abs() <= 2**-7 * want.abs() + 2**-8 * (z * v).abs() + 1e-6).all()

"""A row alone has the bits that it has beside others, from 148 groups of 16 weight rows on (B200 only)."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _bf16(shape, seed, std=1.0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape, device="cuda", generator=gen) * std).to(torch.bfloat16)


@pytest.mark.parametrize("N,same", [(2352, False), (2353, True), (2368, True), (6151, True)])  # 147 and 148 groups, a ragged last one
@pytest.mark.parametrize("K", [72, 2048, 6144])
def test_projection(native_lib, N, same, K):
    n = native_lib
    x, w = _bf16((3, K), K), _bf16((N, K), N, 0.1)
    one, three = torch.full((1, N), float("nan"), device="cuda"), torch.full((3, N), float("nan"), device="cuda")
    n.skinny_bf16(x, w, three, n.SK_OUT_F32)
    for r in range(3):
        n.skinny_bf16(x[r : r + 1], w, one, n.SK_OUT_F32)
        # otherwise: other sums of the same products, 2^-23 an addition
        assert torch.equal(one[0], three[r]) if same else ((one[0] - three[r]).abs() <= (K / 8 + 32) * 2.0**-23 * (x[r].float().abs() @ w.float().abs().T)).all()
    best = torch.zeros(1, dtype=torch.int64, device="cuda")
    n.skinny_bf16(x[2:], w, best, n.SK_OUT_ARGMAX_F32, N=N, channel=5, os_=0)
    assert 0xFFFFFFFF - (int(best) & 0xFFFFFFFF) == int(one.argmax()) + 5


@pytest.mark.parametrize("N,F,K", [(24, 8, 72), (3072, 8192, 2048), (1000, 0, 512), (40, 1200, 264)])
def test_dual_and_gated_projection(native_lib, N, F, K):
    n = native_lib
    x1, x2, w, gu = _bf16((2, K), 1), _bf16((2, K), 2), _bf16((N, K), 3, K**-0.5), _bf16((2 * max(F, 1), K), 4, K**-0.5)
    results = []
    for rows in (1, 2):
        out, act = torch.zeros((rows, N), dtype=torch.bfloat16, device="cuda"), torch.zeros((rows, max(F, 1)), dtype=torch.bfloat16, device="cuda")
        if F:
            n.dual_proj(x1[:rows], w, out, x2[:rows], gu[:F], gu[F:], act, n.GLU_GELU_TANH)
        else:
            n.dual_proj(x1[:rows], w, out)
        results.append((out[0].clone(), act[0].clone()))
    assert all(torch.equal(a, b) for a, b in zip(*results))
    if F >= 148 * 8:
        acts = [torch.zeros((rows, F), dtype=torch.bfloat16, device="cuda") for rows in (1, 2)]
        for act in acts:
            n.skinny_bf16_swiglu(x2[: act.shape[0]], gu[:F], gu[F:], act)
        assert torch.equal(acts[0][0], acts[1][0])

"""Projections of one to eight rows, dense and gated: mma.sync from two rows on, FMAs for one row and for few outputs."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _bf16(shape, seed, std=1.0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape, device="cuda", generator=gen) * std).to(torch.bfloat16)


def _bound(x, w):
    """Of fp32 sums of exact bf16 products in any order, each addition off by at most a unit in the last place (the tensor core truncates)."""
    return (x.shape[-1] / 8 + 32) * 2.0**-23 * (x.double().abs() @ w.double().abs().T)


# groups of 16 outputs around what the kernels take (63 fall to the FMA kernel), ragged N, the two depths (296 groups, more), ragged K
@pytest.mark.parametrize("rows", [1, 2, 5, 8])
@pytest.mark.parametrize("N,K", [(1008, 256), (1009, 64), (1031, 200), (4736, 72), (4744, 4104), (6144, 2056)])
def test_projection_against_64_bits(rows, N, K):
    from glm_tpu_b200.ops import native as n

    x, w = _bf16((rows, K), rows + K), _bf16((N, K), N, 0.1)
    out = torch.full((rows, N), float("nan"), device="cuda")
    n.skinny_bf16(x, w, out, n.SK_OUT_F32)
    want = x.double() @ w.double().T
    assert ((out.double() - want).abs() <= _bound(x, w)).all()
    if N > 1008 and rows > 2:  # a row's bits do not depend on its neighbours (two rows and more)
        pair = torch.full((2, N), float("nan"), device="cuda")
        n.skinny_bf16(x[rows - 2 :], w, pair, n.SK_OUT_F32)
        assert torch.equal(pair, out[rows - 2 :])
    best = torch.zeros(rows, dtype=torch.int64, device="cuda")
    n.skinny_bf16(x, w, best, n.SK_OUT_ARGMAX_F32, N=N, channel=7, os_=0)
    token = 0xFFFFFFFF - (best & 0xFFFFFFFF)
    assert torch.equal(token, out.argmax(dim=1) + 7)


@pytest.mark.parametrize("rows,N,K", [(1, 512, 264), (3, 509, 4104), (8, 2376, 128), (8, 504, 128)])
def test_gated_projection(rows, N, K):
    from glm_tpu_b200.ops import native as n

    x, wg, wu = _bf16((rows, K), 3), _bf16((N, K), 4, 0.1), _bf16((N, K), 5, 0.1)
    act = torch.full((rows, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    n.skinny_bf16_swiglu(x, wg, wu, act)
    g, u = (x.float() @ wg.float().T).bfloat16().float(), (x.float() @ wu.float().T).bfloat16().float()
    want = g * torch.sigmoid(g) * u
    # either factor may land on the neighbouring bf16 (2^-8), the gate's slope is at most 1.1, and the result is rounded once more
    assert ((act.float() - want).abs() <= 2**-6 * want.abs() + 2**-8 * u.abs() * 1.1 * g.abs().clamp_min(2**-8)).all()


@pytest.mark.parametrize("rows", [1, 2, 8])
@pytest.mark.parametrize("N,K", [(1009, 200), (2048, 2048), (6144, 6144), (6144, 16384)])
@pytest.mark.parametrize("sign", [0, 1])
def test_sums_are_as_exact_as_fp32_additions(rows, N, K, sign):
    """2-norm of the error: whatever K is, about that of a few additions."""
    from glm_tpu_b200.ops import native as n

    x, w = _bf16((rows, K), rows + K), _bf16((N, K), N, 0.1)
    if sign:  # nothing cancels: an accumulator that truncates loses something in every step
        x, w = x.abs(), w.abs()
    out = torch.empty(rows, N, device="cuda")
    n.skinny_bf16(x, w, out, n.SK_OUT_F32)
    want = x.double() @ w.double().T
    err = float((out.double() - want).norm() / want.norm())
    # parts of n random products out of K are off by u sqrt(n / K) of the result when added, u = 2^-24 / sqrt(3) at most: eight warps in pairs 3 u^2, a warp's own
    # sum 1, the four sums of a chunk 2.5 (where nothing cancels the parts are n / K, less); sixteen products alone are truncated, 2^-24
    assert err <= 2.0**-24 * (1 + (6.5 / 3) ** 0.5)

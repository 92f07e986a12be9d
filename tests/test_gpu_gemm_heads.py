"""Per-head products in one launch of the persistent tcgen05 GEMM, with the second operand as it lies: [N, K] or [K, N] per head."""

import pytest
import torch

pytestmark = pytest.mark.gpu


# one tile, ragged rows, several column blocks, more tiles than CTAs; the operand's rows begin and end inside a larger table
@pytest.mark.parametrize("rows,heads,N,K,lead,tail", [(1, 1, 64, 64, 0, 0), (130, 3, 512, 192, 0, 40), (300, 8, 264, 128, 24, 8), (700, 64, 256, 512, 192, 0)])
@pytest.mark.parametrize("by_k", [True, False])
def test_against_fp32(native_lib, rows, heads, N, K, lead, tail, by_k):
    gen = torch.Generator(device="cuda").manual_seed(rows + N)
    bf = lambda *s: (torch.randn(*s, device="cuda", generator=gen) * 0.5).to(torch.bfloat16)  # noqa: E731
    a, b = bf(rows, heads, K), bf(heads, lead + (K if by_k else N) + tail, N if by_k else K)
    wide = torch.full((rows, heads, N + 64), float("nan"), dtype=torch.bfloat16, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    native_lib.gemm_bf16_heads(a, b, lead, by_k, wide, N=N, K=K, status=status)
    torch.cuda.synchronize()
    part = b[:, lead : lead + (K if by_k else N)].double()
    want = torch.einsum("rhk,hkn->rhn" if by_k else "rhk,hnk->rhn", a.double(), part)
    size = torch.einsum("rhk,hkn->rhn" if by_k else "rhk,hnk->rhn", a.double().abs(), part.abs())
    assert int(status) == 0 and wide[..., N:].isnan().all()
    assert ((wide[..., :N].double() - want).abs() <= 2**-8 * want.abs() + 1e-5 * size).all()

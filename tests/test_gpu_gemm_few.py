"""Dense GEMM of few rows: weights as M, K dealt to a cluster (B200 only)."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _bf16(shape, seed, std=1.0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape, device="cuda", generator=gen) * std).to(torch.bfloat16)


# one row and one column block more than a tile takes, K with a ragged last step, strided operands and results, blocks of rows, every number of parts
@pytest.mark.parametrize("rows,N,K", [(1, 8, 72), (9, 136, 1032), (16, 256, 576), (100, 1000, 2056), (128, 264, 4096), (129, 384, 1096), (256, 128, 1600)])
@pytest.mark.parametrize("splits", [0, 1, 2, 3, 4, 6, 8])
def test_few_rows_against_64_bits(native_lib, rows, N, K, splits):
    n = native_lib
    a, b = _bf16((rows, K + 16), rows + K)[:, 8 : 8 + K], _bf16((N, K + 8), N, 0.1)[:, :K]
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    outs = [torch.full((rows, N + 8), float("nan"), dtype=dtype, device="cuda")[:, :N] for dtype in (torch.float32, torch.bfloat16, torch.float32)]
    parts = -(-(K // 64 + (K % 64 > 0)) // max(splits, 1))
    n.lib().glmb_set_gemm_variant(16 + splits)
    try:
        if splits and parts * (splits - 1) >= -(-K // 64):  # a part would be empty: another form takes it
            n.lib().glmb_set_gemm_variant(0)
        for out in outs:
            n.gemm_bf16_tc(a, b, out, status=status)
    finally:
        n.lib().glmb_set_gemm_variant(0)
    assert int(status) == 0
    want, size = a.double() @ b.double().T, a.double().abs() @ b.double().abs().T
    # the tensor core truncates as it adds sixteen products at a time: an ulp a step at most; the parts' sums are rounded
    assert ((outs[0].double() - want).abs() <= (K / 16 + 16) * 2.0**-23 * size).all()
    assert torch.equal(outs[1], outs[0].to(torch.bfloat16)) and torch.equal(outs[0], outs[2])


@pytest.mark.parametrize("rows", [9, 60, 128, 129, 200, 256, 257])
@pytest.mark.parametrize("N,K", [(256, 6144), (2048, 2048), (4096, 18432), (6144, 4096)])
def test_chosen_form_is_as_exact_as_the_others(native_lib, rows, N, K):
    """Error against 64 bits (2-norm) of the form that is chosen and of pairs of SMs, which add all of K in the tensor core."""
    n = native_lib
    a, b = _bf16((rows, K), rows), _bf16((N, K), N, K**-0.5)
    out = torch.empty((rows, N), device="cuda")
    want = a.double() @ b.double().T
    errors = []
    for variant in (0, 256):
        n.lib().glmb_set_gemm_variant(variant)
        try:
            n.gemm_bf16_tc(a, b, out)
        finally:
            n.lib().glmb_set_gemm_variant(0)
        errors.append(float((out.double() - want).norm() / want.norm()))
    assert errors[0] <= 1.02 * errors[1], errors

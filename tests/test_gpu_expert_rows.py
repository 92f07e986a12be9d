"""Routed experts of one to eight rows: an expert's weights are read once for all rows that chose it."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _bf16(shape, seed, std=1.0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape, device="cuda", generator=gen) * std).to(torch.bfloat16)


# one row, shared and repeated experts, as many routes as the kernels take, a single channel group, ragged output columns
@pytest.mark.parametrize("rows,top,E,F,K,N", [(1, 4, 6, 64, 200, 40), (8, 4, 9, 72, 136, 48), (5, 3, 3, 1536, 1024, 130), (8, 32, 40, 8, 8, 16), (2, 1, 1, 520, 64, 16)])
def test_experts_shared_by_rows(native_lib, rows, top, E, F, K, N):
    n = native_lib
    gen = torch.Generator().manual_seed(rows * 100 + top)
    ids = torch.stack([torch.randint(0, E, (top,), generator=gen) for _ in range(rows)]).to(torch.int32)  # a row may name an expert twice
    bad = ids.clone()
    bad[0, 0] = E + 4  # clamped to the last expert and reported
    weights = (torch.rand(rows, top, generator=gen) + 0.1).cuda()
    x, gate_up, down = _bf16((rows, K), 1), _bf16((E, 2 * F, K), 2, K**-0.5), _bf16((E, N, F), 3, F**-0.5)
    for given, clamped, flag in ((ids, ids, 0), (bad, bad.clamp(max=E - 1), n.STATUS_BAD_INDEX)):
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        act = torch.full((rows * top, F), float("nan"), dtype=torch.bfloat16, device="cuda")
        n.expert_glu(x, given.cuda(), weights, gate_up, act, n.GLU_SILU, status=status)
        out = torch.full((rows, N), float("nan"), device="cuda")
        n.expert_down(act, given.cuda(), down, out)
        torch.cuda.synchronize()
        assert int(status) == flag
        for r in range(rows):
            total, limit = (torch.zeros(N, dtype=torch.float64, device="cuda") for _ in range(2))
            for s in range(top):
                e, a = int(clamped[r, s]), act[r * top + s]
                z = (gate_up[e].double() @ x[r].double()) * float(weights[r, s])
                want = z[:F] * torch.sigmoid(z[:F]) * z[F:]
                assert ((a.double() - want).abs() <= 2**-8 * want.abs() + 1e-5).all(), (r, s)
                total += down[e].double() @ a.double()
                # fp32 sums of exact bf16 products, each addition off by at most a unit in the last place
                limit += (F / 8 + 32) * 2.0**-23 * (down[e].double().abs() @ a.double().abs()) + 2.0**-22 * (down[e].double() @ a.double()).abs()
            assert ((out[r].double() - total).abs() <= limit + 2.0**-22 * total.abs()).all(), r

"""Experts on 8-route tiles, the tcgen05 form that short prefill chunks take, against a plain restatement (B200 only)."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# K a multiple of 128 and not, column blocks with a ragged end, experts of one route, of more than 64 (several pieces) and of none, other GPUs' experts, a tile
# list without a count on the device
@pytest.mark.parametrize("rows,tk,E,ebase,el,H,I,skew,counted", [
    (1, 2, 8, 0, 8, 512, 512, 0.0, True), (9, 4, 8, 0, 8, 640, 576, 0.0, False), (200, 8, 16, 4, 9, 576, 640, 0.0, True),
    (256, 2, 12, 0, 12, 1088, 528, 3.0, True), (33, 8, 64, 32, 32, 512, 1024, 1.0, True),
])
def test_tiles_of_eight_on_tcgen05(native_lib, rows, tk, E, ebase, el, H, I, skew, counted):
    from glm_tpu_b200.models.glm_moe_dsa.weights import quantize_fp8
    from glm_tpu_b200.oracle.contract import dequantize_fp8

    n = native_lib
    gen = torch.Generator().manual_seed(rows + H + I)
    x = (torch.randn(rows, H, generator=gen) * 0.5).to(torch.bfloat16)
    odds = torch.arange(1, E + 1, dtype=torch.float32) ** -skew
    ids = torch.multinomial(odds.expand(rows, E), tk, replacement=False, generator=gen).to(torch.int32)
    weight = torch.rand(rows, tk, generator=gen) + 0.1
    (wg, sg), (wu, su) = (quantize_fp8(torch.randn(el, I, H, generator=gen) * 0.05, (128, 128), gen) for _ in range(2))
    wd, sd = quantize_fp8(torch.randn(el, H, I, generator=gen) * 0.05, (128, 128), gen)
    P = rows * tk
    tiles = P // 8 + el
    d = lambda t: t.to(DEV).contiguous()  # noqa: E731
    expert, routes, count = torch.full((tiles,), -7, dtype=torch.int32, device=DEV), torch.full((tiles, 8), -7, dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    n.route_sort8(d(ids), ebase, el, expert, routes, count, torch.empty(P, dtype=torch.int32, device=DEV))
    counter = count if counted else None  # tiles past the last one belong to no expert
    x_d, w_d = d(x), d(weight)
    gate, up, down = (d(wg), d(sg)), (d(wu), d(su)), (d(wd), d(sd))
    results = []
    for mma in (1, 0):  # this form, then the fp32 kernels
        n.set_moe_mma(mma)
        act = torch.full((P, I), float("nan"), dtype=torch.bfloat16, device=DEV)
        dw = torch.full((P, H), float("nan"), dtype=torch.bfloat16, device=DEV)
        n.moe_gateup_fp8(x_d, tk, expert, routes, counter, tiles, 8, gate[0], up[0], gate[1], up[1], ebase, act)
        n.moe_down_fp8(act, w_d, expert, routes, counter, tiles, 8, down[0], down[1], ebase, dw)
        results.append((act.cpu().float(), dw.cpu().float()))
    n.set_moe_mma(1)
    bf = lambda t: t.to(torch.bfloat16).float()  # noqa: E731
    dq = [dequantize_fp8(w, s, (128, 128)).float() for w, s in ((wg, sg), (wu, su), (wd, sd))]
    own = (ids.reshape(-1) >= ebase) & (ids.reshape(-1) < ebase + el)
    for act, dw in results:
        assert bool(act[~own].isnan().all()) and bool(dw[~own].isnan().all())  # other GPUs' routes are not written
        for p in own.nonzero().flatten().tolist():
            e = int(ids.reshape(-1)[p]) - ebase
            g, u = bf(x[p // tk].float() @ dq[0][e].T), bf(x[p // tk].float() @ dq[1][e].T)
            want = g * torch.sigmoid(g) * u
            # either factor may land on the neighbouring bf16 (2^-8 of it), the gate's slope is at most 1.1, and the result is rounded once more
            assert bool(((act[p] - want).abs() <= 2**-6 * want.abs() + 2**-8 * 1.1 * (g * u).abs() + 1e-6).all()), p
            want = bf(act[p] @ dq[2][e].T) * bf(weight.reshape(-1)[p])
            size = (act[p].abs() @ dq[2][e].abs().T) * weight.reshape(-1)[p]
            # the sum may round to the neighbouring bf16 (a step is at most 2^-7 of the value), and its product with the weight is rounded (2^-8)
            assert bool(((dw[p] - want).abs() <= (2**-7 + 2**-8 + 2**-14) * want.abs() + I * 2.0**-24 * size).all()), p


# the shapes above are small: left to its rule the library takes mma.sync for some of them
@pytest.mark.parametrize("case", test_tiles_of_eight_on_tcgen05.pytestmark[0].args[1])
def test_tiles_of_eight_wherever_they_can(native_lib, case):
    class Forced:
        def __getattr__(self, name):
            return getattr(native_lib, name)

        def set_moe_mma(self, enabled):
            native_lib.set_moe_mma(2 if enabled else 0)

    try:
        test_tiles_of_eight_on_tcgen05(Forced(), *case)
    finally:
        native_lib.set_moe_mma(1)


def test_a_lost_wait_has_the_runners_status_word(native_lib, monkeypatch):
    """The kernels of the 8-route tiles give up their waits after a limit: both launches of a prefill chunk hand over the word that the host reads after it."""
    from glm_tpu_b200.config.model import small_geometry
    from glm_tpu_b200.ops import native
    from glm_tpu_b200.runner.gpu_runner import build_runner

    handed = []

    class Seen:
        def __getattr__(self, name):
            fn = getattr(inner, name)
            if name not in ("glmb_moe_gateup_fp8", "glmb_moe_down_fp8"):
                return fn
            return lambda *args: (handed.append((name, getattr(args[-2], "value", args[-2]))), fn(*args))[1]

    prompt = torch.randint(0, small_geometry(4).vocab_size, (60,), generator=torch.Generator().manual_seed(1)).tolist()
    runner = build_runner(small_geometry(4), world=1, rank=0, device="cuda:0", seed=0, context_capacity=512, lanes=1, use_graphs=False, prefill_chunk=64)
    try:
        runner.model.few_routes_limit = 1 << 20  # 8-route tiles, whatever the small model's count of experts
        inner = native.lib()
        monkeypatch.setattr(native, "_lib", Seen())
        runner.open_lane(0)
        runner.extend(0, prompt)
    finally:
        monkeypatch.setattr(native, "_lib", inner)
        runner.close()
    assert {name for name, _ in handed} == {"glmb_moe_gateup_fp8", "glmb_moe_down_fp8"}
    assert all(word == runner.peer.status_ptr for _, word in handed)

"""Which kernels a prefill chunk's routed experts take."""

import pytest
import torch

from glm_tpu_b200.config.model import small_geometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,grouped", [(256, False), (257, True)])
def test_long_chunks_take_the_grouped_kernel(native_lib, rows, grouped):
    from glm_tpu_b200.runner.gpu_runner import build_runner

    prompt = torch.randint(0, small_geometry(4).vocab_size, (rows,), generator=torch.Generator().manual_seed(rows)).tolist()
    runner = build_runner(small_geometry(4), world=1, rank=0, device="cuda:0", seed=0, context_capacity=512, lanes=1, use_graphs=False, prefill_chunk=320)
    try:
        runner.model.few_routes_limit = 1 << 20  # few routes per expert, whatever the small model's count of experts
        with native_lib.kernel_timeline() as tl:
            runner.prefill(0, prompt)
        names = [name for name, _, _ in tl.rows()]
        assert ("moe_grouped_fp8w" in names) == grouped and ("moe_gateup_fp8" in names) != grouped
        runner.peer.check_status()
    finally:
        runner.close()


@pytest.mark.parametrize("limit,rows,grouped", [("1000000", 257, False), ("1000000", 320, False), ("0", 200, True)])
def test_a_limit_of_the_users_holds_for_every_chunk(native_lib, monkeypatch, limit, rows, grouped):
    from glm_tpu_b200.runner.gpu_runner import build_runner

    monkeypatch.setenv("GLM_B200_FEW_ROUTES", limit)
    prompt = torch.randint(0, small_geometry(4).vocab_size, (rows,), generator=torch.Generator().manual_seed(rows)).tolist()
    runner = build_runner(small_geometry(4), world=1, rank=0, device="cuda:0", seed=0, context_capacity=512, lanes=1, use_graphs=False, prefill_chunk=320)
    try:
        with native_lib.kernel_timeline() as tl:
            runner.prefill(0, prompt)
        names = [name for name, _, _ in tl.rows()]
        assert ("moe_grouped_fp8w" in names) == grouped and ("moe_gateup_fp8" in names) != grouped
        runner.peer.check_status()
    finally:
        runner.close()

"""Logits of given text at places out of order, chosen twice, beside each other and spread over several passes (B200 only)."""

import pytest
import torch

from tests.test_gpu_lane_count import _geometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family", ["glm", "namizen", "zikevik"])
def test_places_in_any_order_are_those_asked_for_one_at_a_time(native_lib, family):
    from glm_tpu_b200.runner.gpu_runner import build_runner

    g = _geometry(family)
    text = torch.randint(0, g.vocab_size, (200,), generator=torch.Generator().manual_seed(7)).tolist()
    runner = build_runner(g, seed=0, device="cuda:0", context_capacity=1024, lanes=1, prefill_chunk=64)

    def logits(want):
        runner.open_lane(0)
        return torch.as_tensor(runner.extend(0, text, want=want))

    try:
        # passes of 64 rows: the third has no place, the first a place twice, the second and last neighbours in order and reversed
        for want in ([70, 3, 195, 5, 3, 196, 71], [196, 195, 71, 70, 5, 3], [63, 64], [199], [0, 1, 2, 3]):
            got = logits(want)
            assert got.shape == (len(want), g.vocab_size) and got.dtype == torch.float32 and got.device.type == "cpu"
            for row, place in zip(got, want):
                assert torch.equal(row, logits([place])[0]), (want, place)
        assert logits([]).shape == (0, g.vocab_size)
        with pytest.raises(ValueError):
            logits([200])
    finally:
        runner.close()

"""A request's logits do not depend on how many other lanes its runner has (two to eight in all), nor on what they hold: bit for bit, in every family."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _geometry(family):
    if family == "glm":
        from glm_tpu_b200.config.model import glm53_geometry

        return glm53_geometry().truncated(4)
    size = dict(width=2048, heads=16, head_dim=128, vocab=8192)
    if family == "namizen":
        from glm_tpu_b200.config.namizen import bench_namizen

        return bench_namizen(2, kv_heads=4, ff=8192, chunk=2048, **size)
    from glm_tpu_b200.config.zikevik import RoutedSpec, bench_zikevik

    return bench_zikevik(3, ff=1536 if family == "routed" else 8192, routed=RoutedSpec(16, 4, 1536) if family == "routed" else None, **size)


@pytest.mark.parametrize("family", ["glm", "namizen", "zikevik", "routed"])
def test_lanes_of_a_runner_do_not_change_the_bits(native_lib, family):
    from glm_tpu_b200.runner.gpu_runner import build_runner

    g = _geometry(family)
    gen = torch.Generator().manual_seed(5)
    texts = [torch.randint(0, g.vocab_size, (n,), generator=gen).tolist() for n in (61, 40, 77, 45)]
    results = []
    for lanes in (2, 4):
        runner = build_runner(g, seed=0, device="cuda:0", context_capacity=1024, lanes=lanes, prefill_chunk=64)
        for lane in range(lanes):
            runner.open_lane(lane)
            runner.extend(lane, texts[lane][:50 if lane == 0 else 30])
        # one wanted place and several of a short stretch, then decoding
        rows = [runner.extend(0, texts[0][50:56], want=[3, 5] if lanes == 2 else [0, 2, 3, 5])[-1]]
        for step in range(4):
            feeds = {lane: texts[lane][56 + step if lane == 0 else 30 + step] for lane in range(lanes)}
            rows.append(runner.decode_logits(feeds)[0])
        results.append(torch.stack([torch.as_tensor(r).cpu() for r in rows]))
        runner.peer.check_status()
        runner.close()
    assert torch.equal(results[0], results[1])


def test_eight_key_heads_on_a_long_ring(native_lib):
    """Decode attention with a part of the keys per CTA (two and four lanes) and with two (five and eight)."""
    from glm_tpu_b200.config.namizen import bench_namizen
    from glm_tpu_b200.runner.gpu_runner import build_runner

    g = bench_namizen(2, kv_heads=8, ff=8192, chunk=4096, width=2048, heads=16, head_dim=128, vocab=8192)
    gen = torch.Generator().manual_seed(9)
    texts = [torch.randint(0, g.vocab_size, (n,), generator=gen).tolist() for n in (1300, 40, 77, 45, 600, 3, 64, 65)]
    results = []
    for lanes in (2, 4, 5, 8):
        runner = build_runner(g, seed=0, device="cuda:0", context_capacity=4096, lanes=lanes, prefill_chunk=512)
        for lane in range(lanes):
            runner.open_lane(lane)
            runner.extend(lane, texts[lane][:-2])
        rows = [runner.decode_logits({lane: texts[lane][step] for lane in range(lanes)}) for step in (-2, -1)]
        results.append(torch.stack([torch.as_tensor(r[lane]).cpu() for r in rows for lane in (0, 1)]))
        runner.peer.check_status()
        runner.close()
    assert all(torch.equal(results[0], r) for r in results[1:])

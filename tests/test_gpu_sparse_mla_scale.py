"""Where sparse attention's output is scaled and divided by other warps and another quotient than a plain loop's (B200 only)."""

import pytest
import torch

from tests.test_gpu_sparse_mla_rows import H, L, W, _case, _exact, _run

pytestmark = pytest.mark.gpu


def test_a_key_chosen_again_and_again_is_returned_to_the_bit(native_lib):
    """All weights are 1 and the sums are exact (8 bits times at most 2,048), so only a correctly rounded quotient gives the key itself."""
    counts = [1, 2, 3, 7, 11, 127, 128, 129, 641, 1021, 1999, 2047, 2048] * 12  # more rows than CTAs
    q, cache, sel, cnt, lane = _case(counts, 2048, 4096, seed=3)
    sel = sel[:, :1].expand(-1, 2048).contiguous()
    out, status = _run(native_lib, q, cache, sel, cnt, lane, 2048, W**-0.5)
    assert status == 0
    assert torch.equal(out, cache[1, 1, sel[:, 0].long(), :L][:, None].expand(-1, H, -1))


@pytest.mark.parametrize("growing", [slice(0, 32), slice(32, 64), slice(5, 6), slice(63, 64)])
def test_maxima_that_grow_for_some_heads_only(native_lib, growing):
    counts = [129, 640, 1024] * 60
    q, cache, sel, cnt, lane = _case(counts, 1024, 2048, seed=6)
    q *= 0.02  # the other heads: scores close to each other, whose maxima hardly move
    q[:, growing] = 2.0
    cache[1, 1] = cache[1, 1].abs() * torch.linspace(0.02, 1.0, 2048, device="cuda")[:, None].to(torch.bfloat16)
    out, status = _run(native_lib, q, cache, sel, cnt, lane, 1024, 0.1)
    assert status == 0
    want = _exact(q, cache, sel, counts, 0.1)
    # weights and result rounded to bf16, as in the test of the rows
    assert float(((out.double() - want).norm(dim=(1, 2)) / want.norm(dim=(1, 2))).max()) < 4.5e-3

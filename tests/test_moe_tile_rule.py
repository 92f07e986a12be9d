"""Which form the experts of a short prefill chunk take (CPU only: the rule runs on the host)."""

import pytest

from glm_tpu_b200.ops import native


# us measured on a B200, mma.sync and tcgen05, of routes dealt at random: experts, top, rows, N, K, mode
@pytest.mark.parametrize("experts,top,rows,N,K,mode,mma,tcgen05", [
    (8, 2, 9, 1024, 1024, 0, 6.0, 13.1), (8, 2, 64, 1024, 1024, 1, 7.2, 14.5), (8, 2, 256, 1024, 1024, 0, 32, 23), (64, 4, 16, 512, 2048, 0, 26, 33.4),
    (64, 4, 256, 512, 2048, 0, 69, 42), (64, 4, 48, 2048, 512, 1, 19.1, 23.1), (16, 4, 9, 640, 576, 1, 3.5, 10.0), (16, 4, 256, 640, 576, 0, 31, 20),
    (256, 8, 12, 256, 6144, 0, 66.6, 84.0), (256, 8, 64, 256, 6144, 0, 151, 122), (32, 8, 9, 2048, 6144, 0, 147, 122), (32, 8, 200, 6144, 2048, 1, 550, 138),
    (256, 8, 60, 2048, 6144, 0, 1115, 920), (256, 8, 60, 6144, 2048, 1, 680, 490), (256, 8, 256, 2048, 6144, 0, 1724, 1160),
])
def test_the_faster_form_is_chosen(experts, top, rows, N, K, mode, mma, tcgen05):
    assert native.moe_tiles8_pays(rows * top // 8 + experts, experts, N, K, mode) == (tcgen05 < mma)


def test_odd_lists_have_an_answer():
    assert not native.moe_tiles8_pays(1, 1, 256, 512, 0) and not native.moe_tiles8_pays(0, 4, 256, 512, 1) and not native.moe_tiles8_pays(5, 0, 256, 512, 1)
    assert native.moe_tiles8_pays(4096, 256, 2048, 6144, 0)

"""Which fp32 products leave cuBLAS: those where the library's kernel was measured ahead or level."""

import pytest

from diff_gpt_b200.model.gpt import own_f32


@pytest.mark.parametrize("M,N,K,ends,own", [
    (100, 256, 64, False, True), (100, 64, 128, True, True), (17, 64, 64, False, True), (400, 512, 64, False, True),
    (2, 512, 512, False, False), (3, 2048, 512, True, False), (8, 256, 256, False, False), (16, 192, 192, False, False),
    (2, 64, 64, False, False), (4, 256, 64, False, False), (5, 256, 64, False, True), (5, 128, 128, False, False), (2, 128, 256, True, False), (5, 256, 512, True, False),
    (2, 256, 64, True, True), (16, 64, 128, True, True), (8, 1024, 256, False, True), (16, 2048, 512, True, True),
    (1, 256, 64, False, True), (1, 64, 128, True, False), (1000, 1024, 64, False, False), (17, 64, 516, False, False),
])
def test_rule_at_its_edges(M, N, K, ends, own):
    assert own_f32(M, N, K, ends) is own

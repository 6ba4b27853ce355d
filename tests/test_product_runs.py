"""Where a swapped product cuts k although nobody downstream adds the runs: on both sides of the rule's line, at sizes where both
sides were measured."""

import pytest

from tandemllm_b200.kernels.tensorcore import swapped_runs


@pytest.mark.parametrize("M,N,K,want", [
    (8, 6144, 4096, 4), (1, 5120, 5120, 4), (32, 9216, 4096, 3), (8, 12288, 4096, 2), (64, 9216, 4096, 3), (37, 6144, 2048, 4),
    (64, 14336, 2048, 1), (33, 12288, 2048, 1), (128, 7680, 4096, 1), (65, 18816, 8192, 1), (16, 18816, 2560, 1),
    (128, 2048, 4096, 10), (33, 1024, 1024, 4), (64, 512, 448, 1), (8, 18944, 4096, 1)])
def test_runs_of_sums_that_nobody_adds(M, N, K, want):
    bn = next(b for b in (16, 32, 64, 128) if b >= M)
    assert swapped_runs(M, N, K, bn, 148, False) == want


@pytest.mark.parametrize("M,N,K,want", [(64, 14336, 2048, 2), (128, 7680, 4096, 3), (37, 18944, 4096, 1), (64, 512, 448, 1), (64, 512, 512, 2)])
def test_runs_of_sums_that_the_consumer_adds(M, N, K, want):
    bn = next(b for b in (16, 32, 64, 128) if b >= M)
    assert swapped_runs(M, N, K, bn, 148, True) == want

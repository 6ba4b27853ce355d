"""Which form a product takes, by sizes alone."""

import pytest

from tandemllm_b200.kernels import ops


@pytest.mark.parametrize("M,N,K,run", [
    (8, 2048, 2048, 0), (9, 2048, 2048, 512), (512, 2048, 2048, 512), (513, 2048, 2048, 0),      # rows
    (150, 255, 2048, 0), (150, 256, 2048, 512), (150, 4097, 2048, 0),                            # outputs
    (150, 2048, 1020, 0), (150, 2048, 1024, 256), (150, 2048, 7168, 1792), (150, 2048, 2052, 544),
    (256, 4096, 4096, 1024), (320, 4096, 4096, 0),                                               # four tiles an SM, five
    # below a k of 2048 only where the runs' CTAs come out even: the other side was measured faster whole
    (192, 2048, 1024, 256), (200, 2048, 1024, 0), (300, 2048, 1024, 256), (400, 2048, 1024, 0), (256, 4096, 1024, 0),
    (512, 1024, 1024, 0), (512, 512, 1024, 256)])
def test_32_bit_products_in_runs_of_k(M, N, K, run, monkeypatch):
    monkeypatch.setattr(ops, "sm_count", lambda: 148)
    assert ops.simt_runs(M, N, K) == run

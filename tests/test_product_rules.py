"""Which form a product or an attention takes, by sizes alone."""

import types

import pytest

from tandemllm_b200.kernels import ops, tensorcore


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


@pytest.mark.parametrize("contexts,window,spans", [
    ([512], 0, (1, 0)), ([600] * 2, 0, (3, 256)), ([600] * 8, 0, (1, 0)), ([1030] * 8, 0, (5, 256)), ([1500] * 23, 0, (1, 0)),
    ([100 + 31 * i for i in range(30)], 0, (1, 0)), ([250 + 77 * i for i in range(30)], 0, (3, 1024)),
    ([600] * 60, 0, (1, 0)), ([3000] * 60, 0, (2, 2048)), ([8192, 8000, 7000, 900], 0, (32, 256)),
    ([201 + 185 * i for i in range(22)], 0, (4, 1024)), ([4000] * 4, 512, (1, 0)), ([4000] * 4, 2000, (16, 256)),
    ([9000] * 148, 0, (1, 0))])                                                 # (the tiles alone fill the GPU)
def test_decode_rows_beside_a_portion_in_spans_of_keys(contexts, window, spans):
    assert tensorcore._row_spans(types.SimpleNamespace(sm_count=148), contexts, 8, window) == spans

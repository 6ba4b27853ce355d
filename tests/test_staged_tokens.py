"""A step's token ids are staged whatever holds them: what numpy takes as whole numbers."""

from array import array

import numpy as np
import pytest
import torch

from tandemllm_b200.engine.step import _append_int32s, _int32s

HOLDERS = [[7, 300], (7, 300), range(7, 10), np.array([7, 300]), np.array([7, 300], dtype=np.uint16), torch.tensor([7, 300]),
           bytearray(b"\x07\x09"), bytearray(8), [np.int64(7), 300], [7.0, 300.0], [torch.tensor(7), 300], [2 ** 31 - 1]]


@pytest.mark.parametrize("tokens", HOLDERS + [array("i", [7, 300]), array("q", [7, 300]), array("d", [7, 300]), []])
def test_token_ids_in_any_holder_behind_those_of_other_requests(tokens):
    """As a step with portions stages them."""
    out, want = array("i", [5]), np.zeros(len(tokens), dtype=np.int32)
    want[:] = tokens
    _append_int32s(out, tokens)
    assert out.typecode == "i" and out.tolist() == [5] + want.tolist()


def test_a_token_id_that_does_not_fit_leaves_the_others_as_they_were():
    out = array("i", [5])
    with pytest.raises(OverflowError):
        _append_int32s(out, [1, 2 ** 31])
    assert out.tolist() == [5]


@pytest.mark.parametrize("tokens", HOLDERS)
def test_token_ids_in_any_holder(tokens):
    host, want = np.zeros(16, dtype=np.int32), np.zeros(16, dtype=np.int32)
    n = len(tokens)
    host[2:2 + n], want[2:2 + n] = _int32s(tokens), tokens
    assert (host == want).all() and host[2:2 + n].any() == any(int(t) for t in tokens)


def test_a_token_id_that_does_not_fit_is_refused():
    with pytest.raises(OverflowError):
        np.zeros(2, dtype=np.int32)[:] = _int32s([2 ** 31, 0])

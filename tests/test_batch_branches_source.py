"""The streams and events of the batched solves' parallel branches belong to the
context: a new batch makes none. (Made per captured graph they were 0.45 ms of a
small batch's first solve, 0.69 ms where it had been 0.25.)"""
import os

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cfdrs_b200", "csrc")


@pytest.mark.parametrize("name", ["batch.cu", "batch_ls.cu", "batch_internal.h"])
def test_batches_make_no_streams(name):
    assert "cudaStreamCreate" not in open(os.path.join(CSRC, name)).read()

"""Streaming encoder: every way the slices of a block and its warps can run out, against the checker."""
import pytest
import torch

import bsipytorch_b200
from test_gpu_ewah import _compare, _structured

pytestmark = pytest.mark.gpu


# one slice, a partial group of 8, two groups, three and a rest; slices that fill the last tile of 32 words or leave one
# word in it; 444 blocks of one group and one slice more (two groups per block, the last block short), three groups
@pytest.mark.parametrize("S,W", [(1, 256), (7, 129), (16, 160), (27, 256), (3553, 129), (7111, 255), (7105, 97), (8881, 65),
                                 (16385, 33), (50, 256)])
def test_encoder_at_block_edges(S, W):
    _compare(_structured(S, W, S + W), 0.5)


# The call returns while the slices are still being read: slices that belong to another stream are not reused until the
# stream of the call is done with them.
def test_slices_of_another_stream_outlive_the_call():
    other = torch.cuda.Stream()
    words = torch.randint(-5, 5, (4096, 64), device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(other):
        bsipytorch_b200.bsi_ops.ewah_encode_words(words, 0.2)
        torch.cuda._sleep(200_000_000)          # a tenth of a second of work behind the encoder
    address = words.data_ptr()
    del words
    again = torch.empty(4096, 64, dtype=torch.int64, device="cuda")
    assert not other.query() and again.data_ptr() != address
    torch.cuda.synchronize()


# Refused calls do not use up the words of host memory the encoder reports through: it still returns without a
# synchronising call of torch's (which the fallback without a word makes).
def test_refused_calls_leave_the_encoder_as_it_was():
    ops = bsipytorch_b200.bsi_ops
    empty, words = torch.zeros(8, 0, dtype=torch.int64, device="cuda"), torch.randint(-5, 5, (64, 64), device="cuda")
    for _ in range(70):
        with pytest.raises(RuntimeError):
            ops.ewah_encode_words(empty, 0.2)
    torch.cuda.set_sync_debug_mode("error")
    try:
        ops.ewah_encode_words(words, 0.2)
    finally:
        torch.cuda.set_sync_debug_mode("default")

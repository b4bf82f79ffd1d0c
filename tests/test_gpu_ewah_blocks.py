"""Streaming encoder: every way the slices of a block and its warps can run out, against the checker."""
import pytest

from test_gpu_ewah import _compare, _structured

pytestmark = pytest.mark.gpu


# one slice, a partial group of 8, two groups, three and a rest; slices that fill the last tile of 32 words or leave one
# word in it; 444 blocks of one group and one slice more (two groups per block, the last block short), three groups
@pytest.mark.parametrize("S,W", [(1, 256), (7, 129), (16, 160), (27, 256), (3553, 129), (7111, 255), (7105, 97), (8881, 65),
                                 (16385, 33), (50, 256)])
def test_encoder_at_block_edges(S, W):
    _compare(_structured(S, W, S + W), 0.5)

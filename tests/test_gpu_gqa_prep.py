"""The preparation of grouped-query attention in its forms (head size, distance of the rotated partner, tokens a block) against the oracle."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
import test_gpu_attention as base  # noqa: E402

pytestmark = pytest.mark.gpu


# 771 tokens: blocks of four tokens with a remainder, then few tokens behind cached ones; the last two rotations have no form of their own
@pytest.mark.parametrize("M1,M2", [(771, 3), (16, 512)])
@pytest.mark.parametrize("nh,nkv,d,rot,gated", [(3, 1, 256, 64, True), (2, 1, 256, 128, False), (2, 2, 256, 256, True), (4, 2, 128, 64, False), (5, 1, 128, 128, True),
                                                (2, 1, 256, 96, False), (2, 2, 128, 32, True)])
def test_preparation(nh, nkv, d, rot, gated, M1, M2):
    base.test_gqa_prefill_matches_oracle_with_chunked_cache(nh, nkv, d, rot, gated, M1, M2)

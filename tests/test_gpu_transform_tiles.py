"""The plane transform on both sides of the rule between the B-resident BF16 x 3
kernel and the streaming TF32 one, and at the edges of the former's tiles."""
import numpy as np
import pytest

from tests.test_gpu_transform import _run


@pytest.mark.gpu
@pytest.mark.parametrize("K,N,planes,R,ldi,ldo", [
    (176, 176, 3, 70, 176, 72),      # the largest square matrix that stays resident
    (177, 177, 3, 70, 180, 72),      # the first that is streamed
    (256, 256, 2, 65, 256, 68),      # the largest
    (250, 112, 2, 65, 252, 68),      # resident with few stages
    (1, 1, 1, 1, 4, 4),              # a single entry: one row pair of one tile
    (16, 16, 1, 64, 16, 64),         # one full tile, one chunk, one accumulator column group
    (17, 17, 2, 32, 20, 32),         # one column past each: the two epilogue halves differ
    (33, 49, 310, 64, 36, 64),       # two tiles per CTA with a remainder, odd column groups
])
def test_transform_tiles(cuda, K, N, planes, R, ldi, ldo):
    err, err32 = _run(K, N, planes, R, ldi, ldo, seed=7 * K + N)
    # 24-bit operands in three slices and an FP32 sum of K products of which
    # the accumulator rounds every one: at most (K + 4) 2^-24 of sum |x b|,
    # which is below 6 times the largest |sum x b| for these sizes (3 for K = 1)
    assert err <= 6 * (K + 4) * 2.0 ** -24, (err, err32)

"""Heads of few rows over wide vocabularies: the fold of the partial statistics around the counts of partials at which a row gets
more threads and at which they stop being held in registers, and sums of split contractions around the size up to which eight
warps share an element, against float64 (torch)."""
import pytest

import test_gpu_small_products as S
from autograd_b200 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [N.AG_CE_3XTF32, N.AG_CE_BF16])
@pytest.mark.parametrize("n,c,v", [(1, 32, 16384), (9, 40, 16385), (17, 32, 32800), (8, 36, 65536), (7, 32, 65537),
                                   (592, 128, 4100), (593, 128, 4100)])
def test_head(n, c, v, precision):
    S.test_head(n, c, v, False, 0, 1.0, precision)


@pytest.mark.parametrize("offset", [0, 4])
@pytest.mark.parametrize("n,k,c", [(1, 4096, 8), (37, 4104, 136), (256, 2048, 296), (257, 2048, 296)])
def test_projection(n, k, c, offset):
    S.test_projection(n, k, c, offset, N.AG_CE_3XTF32)


@pytest.mark.parametrize("precision", [N.AG_CE_3XTF32, N.AG_CE_BF16])
@pytest.mark.parametrize("n,c,v", [(2664, 32, 17000), (2665, 32, 17000), (5032, 32, 50000), (5033, 32, 50000)])
def test_head_of_many_rows(n, c, v, precision):
    """Around the counts of rows up to which a row gets more threads, for partials of one round and of more."""
    S.test_head(n, c, v, False, 0, 1.0, precision)

"""GF(2^128) products of the device at operands that fill the integer product's
bit gaps: dense and periodic bit patterns, through the product tree's output."""
import numpy as np
import pytest

import bitz_b200 as bz
from oracle import ffi as of

pytestmark = pytest.mark.gpu

WORDS = [2**64 - 1, 0x1111111111111111, 0x8888888888888888, 0x7777777777777777,
         0x5555555555555555, 0xeeeeeeeeeeeeeeee, 0xfffffffeffffffff, 0x7fffffff7fffffff]


@pytest.mark.parametrize("a", WORDS)
@pytest.mark.parametrize("b", WORDS)
def test_products_of_dense_patterns(a, b):
    of.lib().o_set_clmul_mode(1)
    images = np.zeros((128, 2), dtype=np.uint64)
    images[0::2] = np.uint64(a)
    images[1::2] = np.uint64(b)
    images[64:, 0] = np.uint64(b)
    cols = np.full((8, 2), 2**64 - 1, dtype=np.uint64)
    cols[1:, 0] = np.array([1, 3, 0x10001, 0xffff, a, b, a ^ b], dtype=np.uint64)
    cols[3:, 1] = np.array([0, 1, 1 << 63, a, b], dtype=np.uint64)
    got = bz.gkr_outputs(images, cols)
    want = of.gkr_outputs(images, cols)
    of.lib().o_set_clmul_mode(0)
    assert np.array_equal(got, want)

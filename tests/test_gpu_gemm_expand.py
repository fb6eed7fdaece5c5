"""Q6_K and IQ4_XS prompts of eight column tiles and more (four where rows are copied one by one), whose operand is expanded once: tile edges, parts of K, chunks of row tiles
and the way back to the unpacking kernel, against the fp64 product of the same quantized operands. (the bound: `gpu_util.check_sums`)"""
import pytest

import arcint_b200 as A
from gpu_util import check_sums as check, normal_data as data

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = A.Context(0)
    yield c
    c.close()


# the last column tile with one column, or whole; one super-block; row tiles with one row or all but one; rows that are no
# multiple of 16 bytes, cut along K (a product of three super-blocks an SM and more)
@pytest.mark.parametrize("t", [A.Q6_K, A.IQ4_XS])
@pytest.mark.parametrize("m,k,n", [(1, 28672, 897), (129, 14336, 1024), (255, 14336, 912), (300, 11008, 449), (128 * 56, 256, 897), (128 * 30, 512, 1032)])
def test_expanded_operand(ctx, t, m, k, n):
    w, x = data(t, m, k, n, 40 + m + n)
    ctx.stats_reset()
    got = ctx.run_mul_mat(t, w, k, x)
    assert ctx.stats().get("gemm_tc", 0) == 1
    check(got, t, w, k, x)


def test_chunks_of_row_tiles(ctx):
    """K = 17408: 21 row tiles fill the expanded operand's scratch, the 22nd makes a second chunk."""
    t, m, k, n = A.Q6_K, 21 * 128 + 60, 17408, 385
    w, x = data(t, m, k, n, 3)
    check(ctx.run_mul_mat(t, w, k, x), t, w, k, x)


@pytest.mark.parametrize("t", [A.Q6_K, A.IQ4_XS])
def test_without_scratch(t):
    """The unpacking kernel takes the product where the scratch (8.7 MB) cannot be had."""
    m, k, n = 1300, 3072, 912
    w, x = data(t, m, k, n, 9)
    with A.Context(0) as c:
        c.scratch_limit(4 << 20)
        got = c.run_mul_mat(t, w, k, x)
    check(got, t, w, k, x)

"""The tensor-core prompt GEMM where its tiles, halves, parts of K and row stagings end, against the
fp64 product of the same quantized operands.

The bound: block dots are exact integers and what is left are f32 sums over the K / 256 super-blocks (K / 32 blocks) of a
row, each of at most three roundings of half an ulp (2^-24) of the running sum, so |error| <= 3 n 2^-24 sum|terms|; the sum of the
absolute terms is taken from the operands."""
import numpy as np
import pytest

import arcint_b200 as A
import oracle as O

pytestmark = pytest.mark.gpu

TYPES = [A.Q4_0, A.Q8_0, A.IQ4_NL, A.Q4_K, A.Q5_K, A.Q6_K, A.IQ4_XS]


@pytest.fixture(scope="module")
def ctx():
    c = A.Context(0)
    yield c
    c.close()


def check(got, t, w, k, x):
    ref = O.mul_mat_f64(t, w, k, x, True)
    block = 32 if t in (A.Q4_0, A.Q8_0, A.IQ4_NL) else 256
    # a bound of the absolute terms of an output: |w| row by |x| column
    wa = np.abs(O.dequantize(t, w, k)).reshape(w.shape[0], k).astype(np.float64)
    if t in (A.Q4_K, A.Q5_K):
        # the scale and the mins term are rounded apart: d sc q + dmin m <= |w| + 2 dmin m, and dmin m is minus the weight of code 0
        zero = w.reshape(w.shape[0], k // 256, -1).copy()
        zero[:, :, 16:] = 0
        wa = wa + 2 * np.abs(O.dequantize(t, zero.reshape(w.shape), k)).reshape(w.shape[0], k)
    terms = np.abs(x.astype(np.float64)) @ wa.T
    bound = 3 * (k // block) * 2.0 ** -24 * terms * 1.02 + 1e-30     # 1.02: the activation's own rounding to 8 bits
    assert np.isfinite(got).all()
    assert (np.abs(got - ref) <= bound).all(), float((np.abs(got - ref) / bound).max())


def data(t, m, k, n, seed):
    rng = np.random.default_rng(seed)
    return O.quantize(t, O.fill_normal(m * k, seed, 0.02).reshape(m, k)), rng.normal(0, 1, size=(n, k)).astype(np.float32)


# one super-block; halves of 16, 32, 48 and 64 columns, the second with one column or none; the second column tile with one
# column; row tiles with one row or all but one; parts of K of unequal length (K = 2816: eleven super-blocks)
@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("m,k,n", [(1, 256, 9), (129, 512, 16), (127, 256, 17), (128, 768, 33), (130, 512, 65), (64, 512, 96), (255, 768, 128),
                                   (128, 512, 129), (300, 2816, 24), (140, 2816, 145)])
def test_tile_edges(ctx, t, m, k, n):
    w, x = data(t, m, k, n, 100 + m + n)
    ctx.stats_reset()
    got = ctx.run_mul_mat(t, w, k, x)
    assert ctx.stats().get("gemm_tc", 0) == 1
    check(got, t, w, k, x)


@pytest.mark.parametrize("t", TYPES)
def test_many_units_per_block(ctx, t):
    """More units than SMs, so the rings run over several units of one block, full and short ones."""
    m, k, n = 128 * 60, 512, 128 * 4 + 20
    w, x = data(t, m, k, n, 7)
    got = ctx.run_mul_mat(t, w, k, x)
    check(got, t, w, k, x)


def test_sums_beyond_24_bits(ctx):
    """Constant activations give the largest super-block sums (up to 256 * 1953 * 127): float rounding, not wrap-around."""
    for t in (A.Q4_K, A.Q5_K):
        w, _ = data(t, 64, 512, 9, 3)
        x = np.ones((9, 512), np.float32)
        check(ctx.run_mul_mat(t, w, 512, x), t, w, 512, x)

"""The tiled quantizers of the prompt GEMMs: directly loaded (below 128 tokens) and staged through shared memory, groups of eight columns with
dead ones, tokens with infinities, NaN, zeros, subnormal and huge values. Expected: the products of the decode path, which quantizes
with the same rule in kernels of its own, where that is finite; a token with a NaN or an infinity leaves the others alone."""
import numpy as np
import pytest

import arcint_b200 as A
from gpu_util import make_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [A.Q4_0, A.Q8_0, A.Q4_K, A.Q5_K, A.Q6_K, A.IQ4_XS])
@pytest.mark.parametrize("n", [9, 33, 127, 128, 161])
def test_special_tokens(t, n):
    m, k = 40, 768
    rng = np.random.default_rng(n)
    w = make_weights(t, m, k, 5 + t)
    x = rng.normal(0, 1, (n, k)).astype(np.float32)
    x[1] = 0
    # subnormal and huge scales; the per-32 rule's own limits: 1 / (amax / 127) has to be finite, and the scale is a half (up to 127 * 65504)
    per256 = t in (A.Q4_K, A.Q5_K, A.Q6_K, A.IQ4_XS)
    x[2] *= 1e-39 if per256 else 1e-36
    x[3] *= 1e30 if per256 else 1e5
    x[4] = np.round(x[4] * 8) / 16 * 127                     # halves: ties of both rounding rules
    x[4, ::32] = 127
    x[5, 300] = np.nan
    x[6, 300] = np.inf
    with A.Context(0) as c:
        got = c.run_mul_mat(t, w, k, x)
        assert c.stats().get("gemm_tc", 0) == 1
        ref = np.concatenate([c.run_mul_mat(t, w, k, x[i:i + 4]) for i in range(0, n, 4)])
    ok = np.ones(n, bool)
    ok[[5, 6]] = False
    scale = np.abs(ref[ok]).max(axis=1, keepdims=True)
    assert np.isfinite(got[ok]).all()
    # f32 sums of at most 24 terms in different orders: 24 ulp of the largest partial sum, taken as 16 times a row's largest result
    assert (np.abs(got[ok] - ref[ok]) <= 24 * 2.0 ** -24 * 16 * scale + 1e-44).all()
    # a NaN's code is 0 in the per-256 form (its block's other values count), and the per-32 form carries it on
    if per256:
        assert np.isfinite(got[5]).all() and np.allclose(got[5], ref[5], rtol=1e-3, atol=1e-4 * np.abs(ref[5]).max())
    else:
        assert np.isnan(got[5]).all()

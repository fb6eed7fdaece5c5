"""Q4_K and Q5_K products of a route, whose blocks take their units one after the other from a counter in device memory that is zero again
when a launch ends: many units of very different width, launched again and replayed; fewer units than blocks. (the bound: `gpu_util.check_sums`)"""
import numpy as np
import pytest

import arcint_b200 as A
from gpu_util import check_sums as check, normal_data as data

pytestmark = pytest.mark.gpu


# 24 experts x 30 row tiles and more than one tile for the busy expert; two units a row tile; one unit more than SMs have blocks
@pytest.mark.parametrize("t", [A.Q4_K, A.Q5_K])
@pytest.mark.parametrize("n_exp,m,k,n_tok,hot", [(24, 128 * 30, 512, 700, 0.5), (2, 128, 768, 256, 0.9), (1, 128 * 149, 256, 256, 0.0)])
def test_units_are_dealt_out_once(t, n_exp, m, k, n_tok, hot):
    rng = np.random.default_rng(n_tok + m)
    w, x = data(t, m * n_exp, k, n_tok, 5)
    ids = rng.integers(0, n_exp, (n_tok, 1)).astype(np.int32)
    ids[rng.random((n_tok, 1)) < hot] = 0
    with A.Context(0) as c:
        dw, dx, di, dy = c.upload(w), c.upload(x), c.upload(ids), c.alloc(n_tok * m * 4)
        ti = A.Tensor.f32(di, [1, n_tok])
        ti.type = A.I32

        def product():
            c.graph_begin()
            c.mul_mat_id(A.Tensor.weights(t, dw, k, m, n_exp), A.Tensor.f32(dx, [k, 1, n_tok]), ti, A.Tensor.f32(dy, [m, 1, n_tok]))

        def result():
            got = c.download(dy, (n_tok, m), np.float32)
            c.upload(np.full((n_tok, m), np.nan, np.float32), dy)
            return got

        c.stats_reset()
        product()
        first = result()
        assert c.stats().get("moe_gemm", 0) == 1
        product()
        assert np.array_equal(result(), first)
        g = c.capture(product)
        for _ in range(2):
            c.graph_launch(g)
            c.sync()
            assert np.array_equal(result(), first)
        c.graph_free(g)
        for p in (dw, dx, di, dy):
            c.free(p)
    for e in range(n_exp):
        tok = np.nonzero(ids[:, 0] == e)[0]
        if len(tok):
            check(first[tok], t, w[e * m:(e + 1) * m], k, x[tok])

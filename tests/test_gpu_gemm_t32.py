"""The per-32 prompt GEMM multiplies the block scales on the tensor core: scales at the ends of fp16, against the int8 arm, which multiplies
them in f32 (the product of two halves is exact either way, so the outputs are the same bits)."""
import numpy as np
import pytest

import arcint_b200 as A
from gpu_util import make_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [A.Q4_0, A.Q8_0, A.IQ4_NL])
@pytest.mark.parametrize("n", [9, 128, 200])
def test_scales_at_the_ends_of_fp16(monkeypatch, t, n):
    m, k = 130, 512
    rng = np.random.default_rng(n)
    w = make_weights(t, m, k, 60 + t).reshape(m, k // 32, -1).copy()
    d = np.array([0x0001, 0x03FF, 0x0400, 0x8001, 0x0000, 0x7BFF, 0xFBFF], np.uint16)        # subnormal, smallest normal, zero, largest
    w[:, :, 0:2] = d[rng.integers(0, len(d), (m, k // 32))][:, :, None].view(np.uint8).reshape(m, k // 32, 2)
    w[3, 5, 0:2] = np.array([0x7C00], np.uint16).view(np.uint8)                              # a row with an infinite scale, one with a NaN
    w[70, 9, 0:2] = np.array([0x7E00], np.uint16).view(np.uint8)
    x = (rng.normal(0, 1, (n, k // 32, 32)) * 10.0 ** rng.integers(-7, 6, (n, k // 32, 1))).astype(np.float32).reshape(n, k)
    x[2, :32] = 1e8                                                                          # a block scale beyond fp16
    x[4, 64:96] = 0
    got = []
    for arm in ("", "1"):
        monkeypatch.setenv("B200Q_TC_I8", arm)
        with A.Context(0) as c:
            got.append(c.run_mul_mat(t, w.reshape(m, -1), k, x))
            assert (c.stats().get("gemm_tc_f16", 0) == 1) == (arm == "")
    rows = np.ones(m, bool)
    rows[[3, 70]] = False
    cols = np.arange(n) != 2
    assert np.isfinite(got[0][np.ix_(cols, rows)]).all()
    assert np.array_equal(got[0], got[1], equal_nan=True)

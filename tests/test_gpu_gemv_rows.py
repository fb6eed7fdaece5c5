"""The decode GEMV over rows that begin inside a 16-byte unit, against the fp64 product of the same quantized operands. (the bound: `gpu_util.check_sums`)"""
import numpy as np
import pytest

import arcint_b200 as A
import oracle as O
from gpu_util import check_sums as check, normal_data as data

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = A.Context(0)
    yield c
    c.close()


# K whose rows are no multiple of 16 bytes, every decode width, a ragged number of rows
@pytest.mark.parametrize("t,k", [(A.Q6_K, 256), (A.Q6_K, 1280), (A.Q6_K, 11008), (A.Q6_K, 17152), (A.IQ4_XS, 768), (A.IQ4_XS, 11008),
                                 (A.Q4_0, 288), (A.Q8_0, 1056), (A.IQ4_NL, 2080)])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 8])
def test_decode_rows_inside_16_byte_units(ctx, t, k, n):
    m = 37
    w, x = data(t, m, k, n, 11 * n)
    check(ctx.run_mul_mat(t, w, k, x), t, w, k, x)


# weights that start inside a 16-byte unit themselves, with padded rows: what each type's lane code takes (an even address, 8
# bytes for IQ4_XS) and what goes through the 2-byte loader (IQ4_XS and Q4_K at an even address)
@pytest.mark.parametrize("t,k,off,pad", [(A.Q6_K, 1280, 2, 6), (A.Q6_K, 2048, 14, 0), (A.Q6_K, 2048, 0, 2), (A.IQ4_XS, 1024, 8, 8), (A.IQ4_XS, 1024, 2, 4),
                                         (A.Q4_K, 512, 2, 0), (A.Q4_K, 512, 16, 8), (A.Q5_K, 256, 4, 2), (A.Q8_0, 256, 6, 10), (A.Q4_0, 512, 2, 2)])
@pytest.mark.parametrize("n", [1, 2, 4, 8])
def test_decode_weights_at_odd_addresses(ctx, t, k, off, pad, n):
    m = 19
    w, x = data(t, m, k, n, 7 * n + off)
    stride = w.shape[1] + pad
    buf = np.full(off + m * stride, 0xA5, np.uint8)
    for r in range(m):
        buf[off + r * stride:off + r * stride + w.shape[1]] = w[r]
    dw, dx, dy = ctx.upload(buf), ctx.upload(x), ctx.alloc(n * m * 4)
    tw = A.Tensor.make(t, [k, m, 1, 1], [A.block_bytes(t), stride, stride * m, stride * m], dw + off)
    ctx.graph_begin()
    ctx.mul_mat(tw, A.Tensor.f32(dx, [k, n]), A.Tensor.f32(dy, [m, n]))
    got = ctx.download(dy, (n, m), np.float32)
    for p in (dw, dx, dy):
        ctx.free(p)
    check(got, t, w, k, x)


@pytest.mark.parametrize("t,k", [(A.Q6_K, 512), (A.IQ4_XS, 256), (A.Q4_0, 320)])
@pytest.mark.parametrize("n_tok", [1, 4, 40])
def test_routed_rows_inside_16_byte_units(ctx, t, k, n_tok):
    m, n_expert, n_used = 5, 7, 3                    # five rows: experts too begin inside 16-byte units
    w, x = data(t, m * n_expert, k, n_tok, 5)
    ids = np.random.default_rng(n_tok).integers(0, n_expert, size=(n_tok, n_used)).astype(np.int32)
    dw, dx, di, dy = ctx.upload(w), ctx.upload(x), ctx.upload(ids), ctx.alloc(n_tok * n_used * m * 4)
    ti = A.Tensor.f32(di, [n_used, n_tok])
    ti.type = A.I32
    ctx.graph_begin()
    ctx.mul_mat_id(A.Tensor.weights(t, dw, k, m, n_expert), A.Tensor.f32(dx, [k, 1, n_tok]), ti, A.Tensor.f32(dy, [m, n_used, n_tok]))
    got = ctx.download(dy, (n_tok, n_used, m), np.float32)
    for p in (dw, dx, di, dy):
        ctx.free(p)
    for e in range(n_expert):
        tok, slot = np.nonzero(ids == e)
        if tok.size:
            check(got[tok, slot], t, w[e * m:(e + 1) * m], k, x[tok])

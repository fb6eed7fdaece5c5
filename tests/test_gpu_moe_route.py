"""The route over one block and over a cluster of eight (from 2048 pairs), the router's selection by keys and the combine of four results a
thread, where each can go wrong: pair counts around the switch and that do not divide by eight, one expert with nearly all pairs, experts
without any, more pairs than a block keeps in registers, logits of infinities and NaN, widths that are no multiple of four."""
import numpy as np
import pytest

import arcint_b200 as A
import oracle as O
from gpu_util import TOL, make_weights, nmse, rel_err
from test_gpu_moe_ffn import run_router
from test_gpu_mul_mat_id import run_id

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = A.Context(0)
    yield c
    c.close()


# (the last: 9375 pairs a block of the cluster, more than the eight a thread that stay in registers)
@pytest.mark.parametrize("n_expert,n_used,n_tok,hot", [(5, 1, 2047, 0.9), (5, 1, 2048, 0.9), (40, 3, 683, 0.5), (300, 7, 1001, 0.3), (1030, 2, 1100, 0.0), (9, 1, 75000, 0.97)])
def test_routes_on_both_sides_of_the_switch(ctx, n_expert, n_used, n_tok, hot):
    t, m, k = A.Q8_0, 8, 32
    rng = np.random.default_rng(n_tok)
    w = np.stack([O.random_blocks(t, m, k, rng) for _ in range(n_expert)])
    ids = rng.integers(0, max(1, n_expert - 3), (n_tok, n_used)).astype(np.int32)         # (the last three experts get no pair)
    ids[rng.random((n_tok, n_used)) < hot] = n_expert // 2
    ids[0, 0], ids[-1, -1] = -7, n_expert + 9                                            # clamped
    x = rng.normal(0, 1, (n_tok, 1, k)).astype(np.float32)
    got, st = run_id(ctx, t, w, m, k, x, ids, 0, n_used)
    assert st["moe_route"] == 1
    ref = O.mul_mat_id(t, w, m, k, x, np.clip(ids, 0, n_expert - 1), f64=True)
    assert rel_err(got.reshape(-1, m), ref.reshape(-1, m)) < TOL


@pytest.mark.parametrize("n_exp,n_used", [(8, 8), (100, 4), (512, 10)])
def test_router_infinities_and_nan(ctx, n_exp, n_used):
    """A NaN is never picked; where nothing is left to pick the id is out of range, as it was with floating-point comparisons."""
    rng = np.random.default_rng(n_exp)
    logits = rng.normal(0, 1, (5, n_exp)).astype(np.float32)
    logits[1, 3] = -np.inf
    logits[2, :] = -np.inf
    logits[2, 1:n_used + 1] = rng.normal(0, 1, min(n_used, n_exp - 1)) if n_used < n_exp else 0.5
    logits[3, 5] = np.nan
    logits[4, :] = np.nan
    ids, w = run_router(ctx, logits, n_used, 6.103515625e-5, np.inf)
    for row in (0, 1, 2):
        want_ids, want_w = O.moe_router(logits[row:row + 1], n_used, 6.103515625e-5, np.inf)
        assert np.array_equal(ids[row], want_ids[0])
        assert np.allclose(w[row], want_w[0], rtol=2e-6, atol=1e-9)
    assert 5 not in ids[3] and (ids[4] == np.iinfo(np.int32).max).all()


# four results a thread (300 tokens of 512 are just enough), a width that is no multiple of four groups of 256, rows of y that are not 16-byte
# aligned, too few tokens
@pytest.mark.parametrize("d_model,n_tok,n_used,pad", [(512, 300, 2, 0), (768, 300, 9, 0), (512, 300, 3, 1), (512, 20, 3, 0)])
def test_combine(ctx, d_model, n_tok, n_used, pad):
    t, n_exp, d_ff = A.Q4_0, 12, 64
    gw = np.stack([make_weights(t, d_ff, d_model, 100 + e) for e in range(n_exp)])
    uw = np.stack([make_weights(t, d_ff, d_model, 200 + e) for e in range(n_exp)])
    dw_ = np.stack([make_weights(t, d_model, d_ff, 300 + e) for e in range(n_exp)])
    rng = np.random.default_rng(d_model + n_tok + pad)
    x = rng.normal(0, 1, (n_tok, d_model)).astype(np.float32)
    logits = rng.normal(0, 1.5, (n_tok, n_exp)).astype(np.float32)
    want, _, _ = O.moe_ffn(t, gw, uw, dw_, d_model, d_ff, x, logits, n_used, 6.103515625e-5, float("inf"))

    def w3(arr, k, m):
        rb = arr.shape[-1]
        return A.Tensor.make(t, [k, m, n_exp, 1], [A.block_bytes(t), rb, rb * m, rb * m * n_exp], ctx.upload(arr))

    ld = d_model + pad
    y = np.full((n_tok, ld), 7.0, np.float32)
    dx, dl, dy = ctx.upload(x), ctx.upload(logits), ctx.upload(y)
    ws = [w3(gw, d_model, d_ff), w3(uw, d_model, d_ff), w3(dw_, d_ff, d_model)]
    Y = A.Tensor.make(A.F32, [d_model, n_tok, 1, 1], [4, 4 * ld], dy)
    ctx.graph_begin()
    ctx.moe_ffn(ws[0], ws[1], ws[2], A.Tensor.f32(dx, [d_model, n_tok]), A.Tensor.f32(dl, [n_exp, n_tok]), n_used, 6.103515625e-5, float("inf"), Y)
    got = ctx.download(dy, (n_tok, ld), np.float32)
    for p in (dx, dl, dy):
        ctx.free(p)
    for w in ws:
        ctx.free(w.data)
    assert nmse(got[:, :d_model], want) < 5e-4
    assert (got[:, d_model:] == 7.0).all()

"""The tensor-core prompt GEMM where its tiles, halves, parts of K and row stagings end, against the
fp64 product of the same quantized operands. (the bound: `gpu_util.check_sums`)"""
import numpy as np
import pytest

import arcint_b200 as A
import oracle as O
from gpu_util import check_sums as check, normal_data as data

pytestmark = pytest.mark.gpu

TYPES = [A.Q4_0, A.Q8_0, A.IQ4_NL, A.Q4_K, A.Q5_K, A.Q6_K, A.IQ4_XS]


@pytest.fixture(scope="module")
def ctx():
    c = A.Context(0)
    yield c
    c.close()


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


# whole column tiles only, cut along K: parts of equal and of unequal length, one row tile and a ragged second one
@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("m,k,n", [(128, 4096, 128), (200, 2816, 256), (129, 11008, 128)])
def test_whole_tiles_cut_along_k(ctx, t, m, k, n):
    w, x = data(t, m, k, n, m + n)
    ctx.stats_reset()
    got = ctx.run_mul_mat(t, w, k, x)
    assert ctx.stats().get("gemm_tc", 0) == 1 and ctx.stats().get("gemm_ksplit", 0) == 1
    check(got, t, w, k, x)


@pytest.mark.parametrize("t", TYPES)
def test_many_units_per_block(ctx, t):
    """More units than SMs, so the rings run over several units of one block, full and short ones."""
    m, k, n = 128 * 60, 512, 128 * 4 + 20
    w, x = data(t, m, k, n, 7)
    got = ctx.run_mul_mat(t, w, k, x)
    check(got, t, w, k, x)


# activations of 300, 450 and 612 blocks of the tiled quantizers, whose threads follow that number: 512 and 256 for Q4_K and Q5_K, 512 for the
# per-32 types from the second, for Q6_K and IQ4_XS in the third; short last column tiles
@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("k,n", [(12800, 700), (12800, 1030), (17408, 1030)])
def test_activations_of_many_blocks(ctx, t, k, n):
    m = 40
    w, x = data(t, m, k, n, 9)
    got = ctx.run_mul_mat(t, w, k, x)
    check(got, t, w, k, x)


# (K = 1280: ten activation stages of the per-32 GEMM a unit, in rings of three and four)
@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("k", [512, 1280])
def test_many_units_of_whole_tiles_per_block(ctx, t, k):
    m, n = 128 * 60, 128 * 4
    w, x = data(t, m, k, n, 8)
    ctx.stats_reset()
    got = ctx.run_mul_mat(t, w, k, x)
    assert ctx.stats().get("gemm_tc", 0) == 1 and ctx.stats().get("gemm_ksplit", 0) == 0
    check(got, t, w, k, x)


def integer_blocks(t, m, nsb, rng, low):
    """Packed super-blocks with d = 1, dmin = 0, every sub-scale 63 and codes low .. top, and the weights as integers [m, 256 nsb]"""
    top = 15 if t == A.Q4_K else 31
    q = rng.integers(low, top + 1, size=(m, nsb, 8, 32)).astype(np.uint8)
    w = np.zeros((m, nsb, A.block_bytes(t)), np.uint8)
    w[:, :, 0:2] = np.frombuffer(np.float16(1).tobytes(), np.uint8)
    w[:, :, 4:8] = 63 | (3 << 6)                            # sub-scales 0..3 and the two high bits of 4..7
    w[:, :, 12:16] = 15                                     # their four low bits
    if t == A.Q5_K:
        w[:, :, 16:48] = ((q >> 4) << np.arange(8, dtype=np.uint8)[None, None, :, None]).sum(2)
    w[:, :, -128:] = ((q[:, :, 0::2] & 15) | ((q[:, :, 1::2] & 15) << 4)).reshape(m, nsb, 128)
    return w.reshape(m, -1), 63.0 * q.reshape(m, -1)


def integer_codes(n, nsb, rng, one_sided):
    """Integer activations whose 8-bit codes are themselves (every super-block holds a 127): [n, 256 nsb]; one_sided[s]: 1 or -1 for codes of
    that sign only, 100 and more, 0 for codes around zero"""
    x = np.empty((n, nsb, 256), np.float32)
    for s in range(nsb):
        x[:, s] = one_sided[s] * rng.integers(100, 128, (n, 256)) if one_sided[s] else rng.integers(-60, 61, (n, 256))
        x[np.arange(n), s, rng.integers(0, 256, n)] = 127 * (one_sided[s] or 1)
    return x.reshape(n, -1)


@pytest.mark.parametrize("t", [A.Q4_K, A.Q5_K])
@pytest.mark.parametrize("n", [9, 40, 128])
@pytest.mark.parametrize("side", [1, -1])
def test_sums_beyond_24_bits(ctx, t, n, side):
    """Integer sums of a super-block past 2^24, with scales of 1. Two exact chains (Q4_K): the sum, rounded once. Four (Q5_K): three
    additions of one sign, each rounded by half an ulp of at most the sum."""
    rng = np.random.default_rng(n)
    w, wi = integer_blocks(t, 130, 1, rng, 12 if t == A.Q4_K else 28)
    x = integer_codes(n, 1, rng, [side])
    exact = x.astype(np.float64) @ wi.T
    assert np.abs(exact).max() > 2 ** 24 and (exact.astype(np.float32) != exact).any()
    got = ctx.run_mul_mat(t, w, 256, x)
    if t == A.Q4_K:
        assert np.array_equal(got, exact.astype(np.float32))
    assert (np.abs(got - exact) <= 3 * 2.0 ** -24 * np.abs(exact)).all()


@pytest.mark.parametrize("t,edge", [(A.Q4_K, 17753), (A.Q5_K, 8590)])
def test_sums_at_24_bits(ctx, t, edge):
    """Either side of the one-sided sum of codes up to which one chain is exact, 2^24 over 63 * 15 and over 63 * 31"""
    rng = np.random.default_rng(5)
    w, wi = integer_blocks(t, 64, 1, rng, 14 if t == A.Q4_K else 30)
    wi[0], w[0] = wi.max(), integer_blocks(t, 1, 1, rng, 15 if t == A.Q4_K else 31)[0]
    for total in (edge - 1, edge, edge + 1):
        x = np.zeros((12, 256), np.float32)
        for c in range(12):
            left = total
            for i in range(256):
                x[c, i] = min(127, left) if i < 255 - c else 0
                left -= int(x[c, i])
            assert left == 0
        x[:, 1:] = rng.permuted(x[:, 1:], axis=1)
        exact = x.astype(np.float64) @ wi.T
        assert exact.max() == total * wi.max()
        assert np.array_equal(ctx.run_mul_mat(t, w, 256, x), exact.astype(np.float32))


@pytest.mark.parametrize("t", [A.Q4_K, A.Q5_K])
@pytest.mark.parametrize("m,n", [(300, 24), (128 * 60, 128 * 4 + 20), (128 * 40, 128 * 4)])
def test_more_chains_over_many_units(ctx, t, m, n):
    """Several chains a super-block over several units of a block, of sums past 2^24 and within it; a rounding of the running sum for
    each chain."""
    rng = np.random.default_rng(m + n)
    sides = [0, 1, 1, 0, -1, 0, 0, 1, -1]
    w, wi = integer_blocks(t, m, len(sides), rng, 10)
    x = integer_codes(n, len(sides), rng, sides)
    exact = x.astype(np.float64) @ wi.T
    terms = sum(np.abs(x[:, 256 * s:256 * s + 256].astype(np.float64) @ wi[:, 256 * s:256 * s + 256].T) for s in range(len(sides)))
    got = ctx.run_mul_mat(t, w, 256 * len(sides), x)
    # (the largest running sum is within the sum of the super-blocks' absolute sums)
    assert (np.abs(got - exact) <= (2 if t == A.Q4_K else 4) * len(sides) * 2.0 ** -24 * terms).all()


@pytest.mark.parametrize("t", [A.Q4_K, A.Q5_K])
def test_more_chains_in_route_tiles(ctx, t):
    n_exp, n_used, m, nsb, n_tok = 4, 2, 256, 2, 150
    rng = np.random.default_rng(8)
    blocks = [integer_blocks(t, m, nsb, rng, 10) for _ in range(n_exp)]
    w, wi = np.stack([b[0] for b in blocks]), np.stack([b[1] for b in blocks])
    x = integer_codes(n_tok, nsb, rng, [1, 0])
    ids = O.route_ids(n_used, n_tok, n_exp, 3)
    k, rb = 256 * nsb, w.shape[-1]
    dw, dx, di, dy = ctx.upload(w), ctx.upload(x), ctx.upload(ids), ctx.alloc(n_tok * n_used * m * 4)
    W = A.Tensor.make(t, [k, m, n_exp, 1], [A.block_bytes(t), rb, rb * m, rb * m * n_exp], dw)
    ctx.stats_reset()
    ctx.graph_begin()
    ctx.mul_mat_id(W, A.Tensor.make(A.F32, [k, 1, n_tok, 1], [4, 4 * k, 4 * k], dx), A.Tensor.make(A.I32, [n_used, n_tok, 1, 1], [4, 4 * n_used], di),
                   A.Tensor.f32(dy, [m, n_used, n_tok]))
    got = ctx.download(dy, (n_tok, n_used, m), np.float32)
    assert ctx.stats().get("moe_gemm", 0) == 1
    exact = np.einsum("tk,tumk->tum", x.astype(np.float64), wi[ids])
    assert np.abs(exact).max() > 2 ** 24
    # the second super-block's sum stays below 2^24: a rounding per chain of the first and one of the total
    assert (np.abs(got - exact) <= 5 * 2.0 ** -24 * (np.abs(exact) + 2.0 ** 24)).all()
    for p in (dw, dx, di, dy):
        ctx.free(p)


@pytest.mark.parametrize("t", [A.Q4_K, A.Q5_K])
def test_pairs_of_an_expert_in_any_order(ctx, t):
    """Several tiles to an expert, one token that needs more than one chain: no token's bits depend on who shares its tile."""
    n_exp, m, k, n_tok = 2, 128, 512, 500
    rng = np.random.default_rng(4)
    w, x = data(t, m * n_exp, k, n_tok, 21)
    x[7] = rng.uniform(0.6, 1, k)
    ids = rng.integers(0, n_exp, (n_tok, 1)).astype(np.int32)
    dw, dx, di, dy = ctx.upload(w), ctx.upload(x), ctx.upload(ids), ctx.alloc(n_tok * m * 4)
    ti = A.Tensor.f32(di, [1, n_tok])
    ti.type = A.I32

    def run(order):
        ctx.upload(x[order], dx)
        ctx.upload(ids[order], di)
        ctx.stats_reset()
        ctx.graph_begin()
        ctx.mul_mat_id(A.Tensor.weights(t, dw, k, m, n_exp), A.Tensor.f32(dx, [k, 1, n_tok]), ti, A.Tensor.f32(dy, [m, 1, n_tok]))
        out = np.empty((n_tok, m), np.float32)
        out[order] = ctx.download(dy, (n_tok, m), np.float32)
        assert ctx.stats().get("moe_gemm", 0) == 1
        return out

    first = run(np.arange(n_tok))
    for _ in range(3):
        assert np.array_equal(run(rng.permutation(n_tok)), first)
    for e in range(n_exp):
        tok = np.nonzero(ids[:, 0] == e)[0]
        check(first[tok], t, w[e * m:(e + 1) * m], k, x[tok])
    for p in (dw, dx, di, dy):
        ctx.free(p)

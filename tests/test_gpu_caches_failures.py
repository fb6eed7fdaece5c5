"""GPU tests of the per-graph caches and of the failure path, through the C ABI.

The caches follow the reference's (marfrit/arcint contrib/llama.cpp/patches/
0000-01-kquant-integer-dpas.patch:670-688 activation conversion, :1264-1287 MoE route): keyed on the
tensor's identity as well as on its buffer, because a graph allocator hands one address to several
tensors in turn. The failure path is exercised in the one allowed form: a bounded wait that runs out
by design, no trap, no fault."""
import numpy as np
import pytest

import arcint_b200 as A
import oracle as O
from gpu_util import TOL, make_weights, rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = A.Context(0)
    yield c
    c.close()


def _x(dev, k, n, ident):
    return A.Tensor.make(A.F32, [k, n, 1, 1], [4, 4 * k], dev, ident)


@pytest.mark.parametrize("t,n", [(A.Q4_0, 1), (A.Q4_0, 5), (A.Q4_K, 3), (A.Q4_0, 40), (A.IQ4_XS, 24)])
def test_two_tensors_at_one_address_in_one_graph(ctx, t, n):
    """Layer L+1's activation lands where layer L's was (same address, shape and generation): with the
    tensors' identities in the descriptors both products must use their own contents."""
    m, k = 256, 1024
    w = make_weights(t, m, k, 300 + t)
    rng = np.random.default_rng(17 + n)
    xa = rng.normal(0, 1, size=(n, k)).astype(np.float32)
    xb = rng.normal(0, 1, size=(n, k)).astype(np.float32)
    dw, dx, dy = ctx.upload(w), ctx.upload(xa), ctx.alloc(n * m * 4)
    W, Y = A.Tensor.weights(t, dw, k, m), A.Tensor.f32(dy, [m, n])
    ctx.stats_reset()
    ctx.graph_begin()
    ctx.mul_mat(W, _x(dx, k, n, 0x1000), Y)
    ga = ctx.download(dy, (n, m), np.float32)
    ctx.mul_mat(W, _x(dx, k, n, 0x1000), Y)                 # the same tensor again: cached
    # (a small per-32 product at one or two columns quantizes inside the GEMV and has no cache entry at all)
    fused = ctx.stats().get("gemv_fused_quant", 0) > 0
    assert ctx.stats().get("act_cache_hit", 0) == (0 if fused else 1)
    ctx.upload(xb, dx)                                      # another tensor of the graph at the same address
    ctx.mul_mat(W, _x(dx, k, n, 0x2000), Y)
    gb = ctx.download(dy, (n, m), np.float32)
    assert ctx.stats().get("act_cache_hit", 0) == (0 if fused else 1)
    assert rel_err(ga, O.mul_mat_f64(t, w, k, xa, True)) < TOL
    assert rel_err(gb, O.mul_mat_f64(t, w, k, xb, True)) < TOL
    for p in (dw, dx, dy):
        ctx.free(p)


def test_two_ids_tensors_at_one_address_in_one_graph(ctx):
    """The route cache: two layers' ids at one address within one generation."""
    t, n_exp, n_used, m, k, n_tok = A.Q4_K, 8, 2, 128, 512, 40
    w = np.stack([make_weights(t, m, k, 400 + e) for e in range(n_exp)])
    rb = w.shape[-1]
    rng = np.random.default_rng(5)
    x = rng.normal(0, 1, size=(n_tok, 1, k)).astype(np.float32)
    ids_a = O.route_ids(n_used, n_tok, n_exp, 11)
    ids_b = np.ascontiguousarray(ids_a[::-1])
    assert not np.array_equal(ids_a, ids_b)
    dw, dx, di, dy = ctx.upload(w), ctx.upload(x), ctx.upload(ids_a), ctx.alloc(n_tok * n_used * m * 4)
    W = A.Tensor.make(t, [k, m, n_exp, 1], [A.block_bytes(t), rb, rb * m, rb * m * n_exp], dw)
    X = A.Tensor.make(A.F32, [k, 1, n_tok, 1], [4, 4 * k, 4 * k], dx, 0x10)
    Y = A.Tensor.f32(dy, [m, n_used, n_tok])

    def ids(ident):
        return A.Tensor.make(A.I32, [n_used, n_tok, 1, 1], [4, 4 * n_used], di, ident)

    ctx.graph_begin()
    ctx.mul_mat_id(W, X, ids(0x20), Y)
    ga = ctx.download(dy, (n_tok, n_used, m), np.float32)
    ctx.upload(ids_b, di)
    ctx.mul_mat_id(W, X, ids(0x30), Y)
    gb = ctx.download(dy, (n_tok, n_used, m), np.float32)
    assert rel_err(ga.reshape(-1, m), O.mul_mat_id(t, w, m, k, x, ids_a, f64=True).reshape(-1, m)) < TOL
    assert rel_err(gb.reshape(-1, m), O.mul_mat_id(t, w, m, k, x, ids_b, f64=True).reshape(-1, m)) < TOL
    for p in (dw, dx, di, dy):
        ctx.free(p)


@pytest.mark.parametrize("t,n", [(A.Q4_K, 2), (A.Q8_0, 33)])
def test_capture_records_its_own_quantizer(ctx, t, n):
    """Warm up, then capture WITHOUT starting a new generation in between, then rewrite the activation:
    the replay must multiply by the new contents, i.e. the quantizer is part of the recorded graph."""
    m, k = 192, 2048
    w = make_weights(t, m, k, 500 + t)
    rng = np.random.default_rng(3)
    xa = rng.normal(0, 1, size=(n, k)).astype(np.float32)
    xb = rng.normal(0, 1, size=(n, k)).astype(np.float32)
    dw, dx, dy = ctx.upload(w), ctx.upload(xa), ctx.alloc(n * m * 4)
    W, X, Y = A.Tensor.weights(t, dw, k, m), A.Tensor.f32(dx, [k, n]), A.Tensor.f32(dy, [m, n])
    ctx.graph_begin()
    ctx.mul_mat(W, X, Y)                                    # warm-up: sizes the scratch, fills the cache
    g = ctx.capture(lambda: ctx.mul_mat(W, X, Y))           # no graph_begin: the capture starts its own generation
    ctx.upload(xb, dx)
    ctx.graph_launch(g)
    got = ctx.download(dy, (n, m), np.float32)
    ctx.graph_free(g)
    assert rel_err(got, O.mul_mat_f64(t, w, k, xb, True)) < TOL
    for p in (dw, dx, dy):
        ctx.free(p)


def test_bounded_wait_runs_out_and_context_survives(ctx):
    """A device-side wait that nothing satisfies gives up after its poll limit, sets the error word and
    returns: b200q_synchronize reports B200Q_TIMEOUT once, and the next product on the same context is right."""
    ctx.sync()
    ctx.check(ctx.L.b200q_debug_wait_timeout(ctx.h, 2000))
    st = ctx.L.b200q_synchronize(ctx.h)
    assert st == A.binding.TIMEOUT
    assert b"gave up" in ctx.L.b200q_last_error(ctx.h)
    assert ctx.L.b200q_synchronize(ctx.h) == A.binding.OK          # the word was cleared
    t, m, k = A.Q4_0, 128, 1024
    w = make_weights(t, m, k, 77)
    x = np.random.default_rng(1).normal(0, 1, size=(2, k)).astype(np.float32)
    assert rel_err(ctx.run_mul_mat(t, w, k, x), O.mul_mat_f64(t, w, k, x, True)) < TOL


def prompt(ctx, t, m, k, n, seed):
    """(weights, activation, tensors, device pointers) of a prompt product"""
    w, x = make_weights(t, m, k, seed), np.random.default_rng(seed).normal(0, 1, size=(n, k)).astype(np.float32)
    p = ctx.upload(w), ctx.upload(x), ctx.alloc(n * m * 4)
    return w, x, (A.Tensor.weights(t, p[0], k, m), A.Tensor.f32(p[1], [k, n]), A.Tensor.f32(p[2], [m, n])), p


@pytest.mark.parametrize("t", [A.Q8_0, A.Q4_K, A.Q6_K])
def test_no_memory_for_the_parts_of_k(t):
    """Without memory for the parts of a product cut along K it runs whole, without an error text, and can be recorded."""
    m, k, n = 512, 4096, 512                                # eight parts of 1 MiB; the activation takes at most 4.4 MB
    with A.Context(0) as ctx:
        ctx.scratch_limit(6 << 20)
        w, x, mm, p = prompt(ctx, t, m, k, n, 600 + t)
        ctx.graph_begin()
        ctx.mul_mat(*mm)
        assert rel_err(ctx.download(p[2], (n, m), np.float32), O.mul_mat_f64(t, w, k, x, True)) < TOL
        assert ctx.stats().get("gemm_ksplit", 0) == 0 and ctx.L.b200q_last_error(ctx.h) == b""
        g = ctx.capture(lambda: ctx.mul_mat(*mm))
        ctx.upload(-x, p[1])
        ctx.graph_launch(g)
        assert rel_err(ctx.download(p[2], (n, m), np.float32), O.mul_mat_f64(t, w, k, -x, True)) < TOL
        ctx.graph_free(g)
        ctx.scratch_limit(0)
        ctx.graph_begin()
        ctx.mul_mat(*mm)
        assert ctx.stats().get("gemm_ksplit", 0) == 1
        assert rel_err(ctx.download(p[2], (n, m), np.float32), O.mul_mat_f64(t, w, k, -x, True)) < TOL


def test_capture_takes_the_parts_that_fit():
    """A recording whose parts would not fit the scratch is accepted with fewer of them."""
    t, k, n = A.Q6_K, 4096, 512
    with A.Context(0) as ctx:
        _, _, small, _ = prompt(ctx, t, 128, k, n, 1)       # eight parts of 256 KiB, and the activation scratch
        w, x, big, p = prompt(ctx, t, 512, k, n, 2)         # eight of 1 MiB
        ctx.graph_begin()
        ctx.mul_mat(*small)
        grown = ctx.stats()["workspace_grow"]
        g = ctx.capture(lambda: ctx.mul_mat(*big))
        ctx.graph_launch(g)
        assert rel_err(ctx.download(p[2], (n, 512), np.float32), O.mul_mat_f64(t, w, k, x, True)) < TOL
        assert ctx.stats()["gemm_ksplit"] == 2 and ctx.stats()["workspace_grow"] == grown
        ctx.graph_free(g)


def test_failed_growth_keeps_the_recorded_block():
    """A recording that adds up its parts in the scratch stays good when a later, larger product finds no memory for its own."""
    t, k, n = A.Q6_K, 4096, 512
    with A.Context(0) as ctx:
        w, x, small, p = prompt(ctx, t, 128, k, n, 1)
        _, _, big, _ = prompt(ctx, t, 512, k, n, 2)
        ctx.graph_begin()
        ctx.mul_mat(*small)
        g = ctx.capture(lambda: ctx.mul_mat(*small))
        grown = ctx.stats()["workspace_grow"]
        ctx.scratch_limit(4 << 20)
        ctx.graph_begin()
        ctx.mul_mat(*big)
        assert ctx.stats()["workspace_grow"] == grown
        ctx.upload(2 * x, p[1])
        ctx.graph_launch(g)
        assert rel_err(ctx.download(p[2], (n, 128), np.float32), O.mul_mat_f64(t, w, k, 2 * x, True)) < TOL
        ctx.graph_free(g)


@pytest.mark.parametrize("t", [A.Q4_0, A.Q8_0, A.Q4_K, A.Q5_K, A.Q6_K, A.IQ4_XS])
@pytest.mark.parametrize("cached", [False, True])
def test_prompt_product_waits_for_its_weights(ctx, t, cached):
    """A kernel that writes the weights late, but lets its dependents start at once: the product behind it uses the new weights, with a
    quantizer of its own in between and without."""
    m, k, n = 384, 2048, 40
    wa, x, (W, X, Y), p = prompt(ctx, t, m, k, n, 700 + t)
    wb = make_weights(t, m, k, 800 + t)
    new = ctx.upload(wb)
    ctx.graph_begin()
    ctx.mul_mat(W, X, Y)
    ctx.sync()
    if not cached:
        ctx.graph_begin()
    hits = ctx.stats().get("act_cache_hit", 0)
    ctx.late_copy(p[0], new, wb.nbytes, 2000)
    ctx.mul_mat(W, X, Y)
    got = ctx.download(p[2], (n, m), np.float32)
    assert ctx.stats().get("act_cache_hit", 0) - hits == cached
    assert rel_err(got, O.mul_mat_f64(t, wb, k, x, True)) < TOL
    for q in p + (new,):
        ctx.free(q)


@pytest.mark.parametrize("what", ["scratch", "buffer"])
def test_optional_scratch_goes_back_to_a_full_device(what):
    """A wide Q6_K product holds an expanded operand and parts of K; where the device is full after it, they make room for the activation of
    another product or a caller's buffer. It counts as a growth, no error text stays, and the wide product runs without them."""
    t, m, k, n = A.Q6_K, 1100, 3072, 1000
    with A.Context(0) as ctx:
        w, x, wide, p = prompt(ctx, t, m, k, n, 1)          # 7.1 MB of operand, 4.4 MB a part, 3.2 MB of activation
        v, y, other, q = prompt(ctx, A.Q4_K, 64, 2048, 1000, 2)      # 4.5 MB of activation
        ctx.expand_limit(96 << 20)
        ctx.graph_begin()
        ctx.mul_mat(*wide)
        st = ctx.stats()
        assert st["gemm_kx"] == 1 and st["gemm_ksplit"] == 1
        held = ctx.scratch_total(0)
        ctx.scratch_total(held)                             # full
        ctx.graph_begin()
        if what == "scratch":
            ctx.mul_mat(*other)
            assert rel_err(ctx.download(q[2], (n, 64), np.float32), O.mul_mat_f64(A.Q4_K, v, 2048, y, True)) < TOL
        else:
            ctx.free(ctx.alloc(4 << 20))
        assert ctx.stats()["workspace_grow"] > st["workspace_grow"] and ctx.L.b200q_last_error(ctx.h) == b""
        left = ctx.scratch_total(0)
        assert left < held - (4 << 20)
        ctx.scratch_total(left + (4 << 20))                 # the wide product finds its own activation's block, but none of the optional ones
        ctx.stats_reset()
        ctx.graph_begin()
        ctx.mul_mat(*wide)
        assert rel_err(ctx.download(p[2], (n, m), np.float32), O.mul_mat_f64(t, w, k, x, True)) < TOL
        st = ctx.stats()
        assert (st["gemm_tc"], st.get("gemm_kx", 0), st.get("gemm_ksplit", 0)) == (1, 0, 0)


@pytest.mark.parametrize("t", [A.Q4_0, A.Q8_0, A.IQ4_NL])
def test_no_memory_for_the_f16_activation(monkeypatch, t):
    """Where only the int8 arm's activation fits (2.3 times smaller, the same bits), the product takes that arm: at once, from its cached
    activation, from a recording, and for route tiles. With room again it is the f16 arm."""
    m, k, n = 192, 2048, 500                                # 32 tiles of 256 weights: 2.8 MB in halves, 1.2 MB in bytes
    monkeypatch.setenv("B200Q_NO_KSPLIT", "1")              # (the limit would change the parts of K as well)
    with A.Context(0) as ctx:
        w, x, mm, p = prompt(ctx, t, m, k, n, 900 + t)
        ctx.scratch_limit(2 << 20)
        ctx.graph_begin()
        ctx.mul_mat(*mm)
        small = ctx.download(p[2], (n, m), np.float32)
        ctx.mul_mat(*mm)
        st = ctx.stats()
        assert (st["gemm_tc"], st.get("gemm_tc_f16", 0), st["act_cache_hit"]) == (2, 0, 1) and ctx.L.b200q_last_error(ctx.h) == b""
        g = ctx.capture(lambda: ctx.mul_mat(*mm))
        ctx.graph_begin()
        ctx.mul_mat(*mm)                                    # (finds no room again, and leaves the recording's block alone)
        assert ctx.stats()["workspace_grow"] == st["workspace_grow"]
        ctx.upload(-x, p[1])
        ctx.graph_launch(g)
        assert rel_err(ctx.download(p[2], (n, m), np.float32), O.mul_mat_f64(t, w, k, -x, True)) < TOL
        ctx.graph_free(g)
        ctx.upload(x, p[1])
        ctx.scratch_limit(0)
        ctx.graph_begin()
        ctx.mul_mat(*mm)
        assert ctx.stats()["gemm_tc_f16"] == 1
        whole = ctx.download(p[2], (n, m), np.float32)
        assert rel_err(whole, O.mul_mat_f64(t, w, k, x, True)) < TOL and np.array_equal(small, whole)
    with A.Context(0) as ctx:                               # a recording that was not run before is refused, although the bytes would fit
        _, _, few, _ = prompt(ctx, t, m, k, 200, 1)
        _, _, mm, _ = prompt(ctx, t, m, k, n, 2)
        ctx.graph_begin()
        ctx.mul_mat(*few)
        with pytest.raises(A.B200QError, match="inside a capture"):
            ctx.capture(lambda: ctx.mul_mat(*mm))
        ctx.graph_begin()
        ctx.mul_mat(*mm)
        assert ctx.stats()["gemm_tc_f16"] == 2
    # four experts of 48 rows, two used of 250 tokens: eight tiles at most
    ids = O.route_ids(2, 250, 4, 3)
    got = []
    for limit in (0, 3 << 20):                              # eight tiles: 5.5 MB in halves, 2.4 MB in bytes
        with A.Context(0) as ctx:
            ctx.scratch_limit(limit)
            dw, dx, di, dy = ctx.upload(w), ctx.upload(x[:250]), ctx.upload(ids), ctx.alloc(500 * 48 * 4)
            rb = w.shape[-1]
            ctx.graph_begin()
            for _ in range(2):
                ctx.mul_mat_id(A.Tensor.make(t, [k, 48, 4, 1], [A.block_bytes(t), rb, rb * 48, rb * 192], dw), A.Tensor.f32(dx, [k, 1, 250]),
                               A.Tensor.make(A.I32, [2, 250, 1, 1], [4, 8], di), A.Tensor.f32(dy, [48, 2, 250]))
            got.append(ctx.download(dy, (500, 48), np.float32))
            st = ctx.stats()
            assert (st["moe_gemm"], st["gemm_tc"], st.get("gemm_tc_f16", 0), st["act_cache_hit"]) == (2, 2, 0 if limit else 2, 1), st
    assert np.isfinite(got[0]).all() and np.array_equal(*got)

"""The products that a ggml backend hands to this library, from one decode call to a long prompt, as measurable cases.

Three kinds, each through the public calls of arcint_b200.Context:

  mul_mat  one MUL_MAT call as a backend's graph walk issues it: new generation, product;
  layer    the seven weight products of a transformer layer (q, k, v over one activation; o; gate, up over one
           activation; down) recorded once and replayed, as a serving loop runs its decode step;
  moe      the mixture-of-experts feed-forward block (router, gate, up, SwiGLU, down, weighted sum), replayed from a
           recording for a decode step, called directly for a prompt.

Weights are N(0, 0.02) quantized to the block format, activations N(0, 1), as everywhere in this repository.
"""
import math
import weakref

import torch

from arcint_b200 import binding as B

TYPES = {"q4_0": B.Q4_0, "q8_0": B.Q8_0, "q4_K": B.Q4_K, "q5_K": B.Q5_K, "q6_K": B.Q6_K, "iq4_nl": B.IQ4_NL, "iq4_xs": B.IQ4_XS}
PER32 = ("q4_0", "q8_0", "iq4_nl")
KVALUES = [-127, -104, -83, -65, -49, -35, -22, -10, 1, 13, 25, 38, 53, 69, 89, 113]
CMIN, CMAX = 6.103515625e-5, float(torch.finfo(torch.float32).max)
MOST_MACS = 17408 * 5120 * 2048


def listed():
    return [
        # the smallest call: one attention projection of a 7B model for one token, where launches and start-up count
        {"name": "decode q4_K 4096x4096", "kind": "mul_mat", "type": "q4_K", "m": 4096, "k": 4096, "n": 1},
        # the LM head for one token: a long stream of weights
        {"name": "decode q6_K head", "kind": "mul_mat", "type": "q6_K", "m": 32000, "k": 4096, "n": 1},
        # one token through a layer of a Llama-2-7B in Q4_0, the repository's decode trace
        {"name": "layer q4_0 b1", "kind": "layer", "type": "q4_0", "down": "q4_0", "d": 4096, "ff": 11008, "n": 1},
        # the same layer in the usual mixed quantization (Q4_K with a Q6_K down projection, rows of 9030 bytes) at the
        # widest verify / small-batch width
        {"name": "layer q4_K/q6_K b8", "kind": "layer", "type": "q4_K", "down": "q6_K", "d": 4096, "ff": 11008, "n": 8},
        # a short prompt or a batch of sequences just past the decode widths
        {"name": "short prompt q4_K x24", "kind": "mul_mat", "type": "q4_K", "m": 11008, "k": 4096, "n": 24},
        # the prefill sizes of the benchmark: 512-token prompt chunks of a 7B model ...
        {"name": "prefill q4_0 4096x4096x512", "kind": "mul_mat", "type": "q4_0", "m": 4096, "k": 4096, "n": 512},
        {"name": "prefill q4_K 11008x4096x512", "kind": "mul_mat", "type": "q4_K", "m": 11008, "k": 4096, "n": 512},
        # ... the down projection with a ragged last chunk and rows that are no multiple of 16 bytes ...
        {"name": "prefill q6_K 4096x11008x333", "kind": "mul_mat", "type": "q6_K", "m": 4096, "k": 11008, "n": 333},
        # ... a diffusion transformer's MLP ...
        {"name": "prefill q8_0 12288x3072x4096", "kind": "mul_mat", "type": "q8_0", "m": 12288, "k": 3072, "n": 4096},
        # ... and the largest product of the benchmark
        {"name": "prefill iq4_xs 17408x5120x2048", "kind": "mul_mat", "type": "iq4_xs", "m": 17408, "k": 5120, "n": 2048},
        # a 512-expert, top-10 mixture-of-experts block for one token and for a prompt
        {"name": "moe decode", "kind": "moe", "type": "q4_K", "d": 2048, "ff": 512, "experts": 512, "used": 10, "n": 1},
        {"name": "moe prompt 2048", "kind": "moe", "type": "q4_K", "d": 2048, "ff": 512, "experts": 512, "used": 10, "n": 2048},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "prefill", "prefill", "layer", "moe"])
    names = list(TYPES)
    if kind in ("decode", "prefill"):
        t = rng.choice(names)
        m = _log(rng, 512, 32000)
        if rng.random() < 0.75:
            m = max(512, m // 64 * 64)                       # most models; the others are odd
        k = 256 * _log(rng, 2, 68)
        if kind == "decode":
            n = rng.randint(1, 8)
            if t in PER32 and rng.random() < 0.25:
                k += 32 * rng.randint(1, 7)                  # rows of whole 32-weight blocks only
        else:
            n = _log(rng, 9, 4096)
            m = max(512, min(m, MOST_MACS // (k * n)))
            n = max(9, min(n, MOST_MACS // (k * m)))
        return {"kind": "mul_mat", "type": t, "m": m, "k": k, "n": n}
    if kind == "layer":
        t = rng.choice(names)
        d = 256 * rng.randint(4, 20)
        down = "q6_K" if t in ("q4_K", "q5_K") and rng.random() < 0.5 else t
        return {"kind": "layer", "type": t, "down": down, "d": d, "ff": 256 * rng.randint(2 * d // 256, 3 * d // 256), "n": rng.randint(1, 8)}
    experts = 1 << rng.randint(3, 9)
    return {"kind": "moe", "type": rng.choice(["q4_0", "q4_K", "q6_K", "iq4_xs"]), "d": 256 * rng.randint(2, 8), "ff": 256 * rng.randint(1, 4),
            "experts": experts, "used": rng.randint(2, min(10, experts)), "n": _log(rng, 1, 2048)}


# ---- quantized weights -----------------------------------------------------------------------------------------------

def _halves(x):
    """float tensor [...] -> its fp16 bytes [..., 2]"""
    return x.half().contiguous().view(torch.uint8).view(*x.shape, 2)


def _signed_max(x):
    return x.gather(-1, x.abs().argmax(-1, keepdim=True)).squeeze(-1)


def _over(a, b):
    """a / b in one rounding (a tensor over a number may be multiplied by its reciprocal)"""
    return torch.div(a if torch.is_tensor(a) else torch.full_like(b, a), b if torch.is_tensor(b) else torch.full_like(a, b))


def _inv(d):
    return torch.where(d != 0, 1.0 / d, torch.zeros_like(d))


def _nearest(x):
    kv = torch.tensor(KVALUES, device=x.device, dtype=torch.float32)
    return torch.bucketize(x, (kv[1:] + kv[:-1]) / 2).to(torch.uint8)


def _quantize(t, x):
    """f32 [rows, k] -> packed blocks [rows, row_bytes] (round to nearest inside each block)"""
    rows, k = x.shape
    if t in PER32:
        b = x.view(rows, k // 32, 32)
        if t == "q8_0":
            d = b.abs().amax(-1) / 127
            q = torch.round(b * _inv(d)[..., None]).to(torch.int8).view(torch.uint8)
        else:
            d = _signed_max(b) / (-8 if t == "q4_0" else -127)
            u = b * _inv(d)[..., None]
            c = torch.clamp(torch.floor(u + 8.5), 0, 15).to(torch.uint8) if t == "q4_0" else _nearest(u)
            q = c[..., :16] | (c[..., 16:] << 4)
        return torch.cat([_halves(d), q], -1).reshape(rows, -1)
    n = rows * (k // 256)
    if t in ("q4_K", "q5_K"):
        b, top = x.reshape(n, 8, 32), 15 if t == "q4_K" else 31
        low = b.amin(-1).clamp(max=0)
        sc = (b.amax(-1) - low) / top
        d, dm = (sc.amax(-1) / 63).half().float(), ((-low).amax(-1) / 63).half().float()
        ls = torch.clamp(torch.round(sc * _inv(d)[:, None]), 0, 63)
        lm = torch.clamp(torch.round(-low * _inv(dm)[:, None]), 0, 63)
        q = torch.clamp(torch.round((b + (dm[:, None] * lm)[..., None]) * _inv(d[:, None] * ls)[..., None]), 0, top).to(torch.uint8)
        ls, lm = ls.to(torch.uint8), lm.to(torch.uint8)
        s = torch.cat([ls[:, :4] | ((ls[:, 4:] >> 4) << 6), lm[:, :4] | ((lm[:, 4:] >> 4) << 6), (ls[:, 4:] & 15) | ((lm[:, 4:] & 15) << 4)], -1)
        parts = [_halves(d), _halves(dm), s]
        if t == "q5_K":
            bit = (q >> 4) << torch.arange(8, device=x.device, dtype=torch.uint8)[None, :, None]
            parts.append(bit.sum(1).to(torch.uint8))
            q = q & 15
        parts.append((q[:, 0::2] | (q[:, 1::2] << 4)).reshape(n, 128))
    elif t == "q6_K":
        b = x.reshape(n, 16, 16)
        sc = _signed_max(b) / -32
        d = (sc.abs().amax(-1) / 127).half().float()
        s = torch.clamp(torch.round(sc * _inv(d)[:, None]), -127, 127)
        q = torch.clamp(torch.round(b * _inv(d[:, None] * s)[..., None]), -32, 31) + 32
        q = q.to(torch.uint8).view(n, 2, 4, 32)
        lo = torch.cat([(q[:, :, 0] & 15) | ((q[:, :, 2] & 15) << 4), (q[:, :, 1] & 15) | ((q[:, :, 3] & 15) << 4)], -1)
        hi = (q[:, :, 0] >> 4) | ((q[:, :, 1] >> 4) << 2) | ((q[:, :, 2] >> 4) << 4) | ((q[:, :, 3] >> 4) << 6)
        parts = [lo.reshape(n, 128), hi.reshape(n, 64), s.to(torch.int8).view(torch.uint8), _halves(d)]
    else:
        b = x.reshape(n, 8, 32)
        sc = _signed_max(b) / -127
        d = (sc.abs().amax(-1) / 31).half().float()
        ls = torch.clamp(torch.round(sc * _inv(d)[:, None]), -31, 31)
        q = _nearest(b * _inv(d[:, None] * ls)[..., None])
        u = (ls + 32).to(torch.int32)
        sh = ((u >> 4) << (2 * torch.arange(8, device=x.device))).sum(-1)
        sh = torch.stack([sh & 255, sh >> 8], -1).to(torch.uint8)
        sl = ((u[:, 0::2] & 15) | ((u[:, 1::2] & 15) << 4)).to(torch.uint8)
        parts = [_halves(d), sh, sl, (q[..., :16] | (q[..., 16:] << 4)).reshape(n, 128)]
    return torch.cat(parts, -1).reshape(rows, -1)


def _weights(t, m, k, g):
    out = torch.empty(m, B.row_bytes(TYPES[t], k), dtype=torch.uint8, device="cuda")
    step = max(1, (1 << 25) // k)
    for r in range(0, m, step):
        n = min(step, m - r)
        out[r:r + n] = _quantize(t, torch.randn(n, k, device="cuda", generator=g) * 0.02)
    return out


def _float_of(b):
    """fp16 bytes [..., 2] -> f64 [...]"""
    return b.contiguous().view(torch.float16).squeeze(-1).double()


def _dequantize(t, w, k):
    """packed rows -> f64 [rows, k], each weight exactly what its block says"""
    rows = w.shape[0]
    kv = torch.tensor(KVALUES, device=w.device, dtype=torch.float64)
    if t in PER32:
        b = w.view(rows, k // 32, -1)
        d, q = _float_of(b[..., :2]), b[..., 2:]
        if t == "q8_0":
            v = q.contiguous().view(torch.int8).double()
        else:
            c = torch.cat([q & 15, q >> 4], -1)
            v = c.double() - 8 if t == "q4_0" else kv[c.long()]
        return (d[..., None] * v).view(rows, k)
    b = w.reshape(rows * (k // 256), -1)
    n = b.shape[0]
    if t in ("q4_K", "q5_K"):
        d, dm, s = _float_of(b[:, 0:2]), _float_of(b[:, 2:4]), b[:, 4:16]
        ls = torch.cat([s[:, :4] & 63, (s[:, 8:] & 15) | ((s[:, :4] >> 6) << 4)], -1).double()
        lm = torch.cat([s[:, 4:8] & 63, (s[:, 8:] >> 4) | ((s[:, 4:8] >> 6) << 4)], -1).double()
        p = b[:, -128:].reshape(n, 4, 32)
        q = torch.stack([p & 15, p >> 4], 2).reshape(n, 8, 32)
        if t == "q5_K":
            q = q | (((b[:, None, 16:48] >> torch.arange(8, device=w.device, dtype=torch.uint8)[None, :, None]) & 1) << 4)
        v = (d[:, None] * ls)[..., None] * q.double() - (dm[:, None] * lm)[..., None]
    elif t == "q6_K":
        l, h, s, d = b[:, :128].reshape(n, 2, 2, 32), b[:, 128:192].reshape(n, 2, 1, 32), b[:, 192:208].contiguous().view(torch.int8), _float_of(b[:, 208:])
        low = torch.cat([l & 15, l >> 4], 2)
        high = (h >> torch.arange(0, 8, 2, device=w.device, dtype=torch.uint8)[None, None, :, None]) & 3
        v = (d[:, None] * s.double())[..., None] * ((low | (high << 4)).reshape(n, 16, 16).double() - 32)
    else:
        d, sh = _float_of(b[:, 0:2]), b[:, 2].int() | (b[:, 3].int() << 8)
        sl = torch.stack([b[:, 4:8] & 15, b[:, 4:8] >> 4], -1).reshape(n, 8).int()
        ls = (sl | (((sh[:, None] >> (2 * torch.arange(8, device=w.device))) & 3) << 4)).double() - 32
        p = b[:, 8:].reshape(n, 8, 16)
        v = (d[:, None] * ls)[..., None] * kv[torch.cat([p & 15, p >> 4], -1).long()]
    return v.reshape(rows, k)


def _activation(t, x):
    """f32 [n, k] -> f64, the values the 8-bit activation of the weight type's form stands for"""
    n, k = x.shape
    if t in PER32:
        b = x.view(n, k // 32, 32)
        d = _over(b.abs().amax(-1), 127.0)
        u = b * torch.where(d != 0, _over(1.0, d), torch.zeros_like(d))[..., None]
        q = torch.trunc(u)
        q = torch.where((u - q).abs() >= 0.5, q + torch.sign(u), q)      # halves away from zero
        return (d.half().double()[..., None] * q.double()).view(n, k)
    b = x.view(n, k // 256, 256)
    top = b.abs().amax(-1)
    iq = torch.where(top > 1e-30, _over(127.0, top), torch.zeros_like(top))
    return (_over(top, 127.0).double()[..., None] * torch.round(b * iq[..., None]).double()).view(n, k)


# ---- the cases -------------------------------------------------------------------------------------------------------

_context = None


def _ctx():
    """one context for the process, as a backend keeps one per device"""
    global _context
    if _context is None:
        _context = B.Context(0)
    return _context


class State:
    pass


def _tensor(x):
    return B.Tensor.f32(x.data_ptr(), list(reversed(x.shape)))


def _products(case):
    """(weight type, rows, k, index of its activation) of a layer's products"""
    t, d, ff = case["type"], case["d"], case["ff"]
    return [(t, d, d, 0)] * 3 + [(t, d, d, 1)] + [(t, ff, d, 2)] * 2 + [(case["down"], d, ff, 3)]


def _inputs(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    s, n = State(), case["n"]
    if case["kind"] == "mul_mat":
        s.w = [_weights(case["type"], case["m"], case["k"], g)]
        s.x = [torch.randn(n, case["k"], device="cuda", generator=g)]
    elif case["kind"] == "layer":
        s.w = [_weights(t, m, k, g) for t, m, k, _ in _products(case)]
        s.x = [torch.randn(n, k, device="cuda", generator=g) for k in (case["d"], case["d"], case["d"], case["ff"])]
    else:
        e, d, ff = case["experts"], case["d"], case["ff"]
        s.w = [_weights(case["type"], e * m, k, g) for m, k in ((ff, d), (ff, d), (d, ff))]
        s.x = [torch.randn(n, d, device="cuda", generator=g)]
        # router logits of a skewed expert popularity, Zipf(1.1), the experts in random order
        rank = torch.randperm(e, device="cuda", generator=g).float()
        s.logits = -1.1 * torch.log(rank + 1) + torch.randn(n, e, device="cuda", generator=g)
    return s


def prepare(case, seed):
    s, c, n = _inputs(case, seed), _ctx(), case["n"]
    xs = [_tensor(x) for x in s.x]
    s.graph = None
    if case["kind"] == "moe":
        e, d, ff, t = case["experts"], case["d"], case["ff"], TYPES[case["type"]]
        s.y = [torch.empty(n, d, device="cuda"), torch.empty(n, case["used"], dtype=torch.int32, device="cuda"), torch.empty(n, case["used"], device="cuda")]
        w = [B.Tensor.weights(t, p.data_ptr(), k, m, e) for p, m, k in zip(s.w, (ff, ff, d), (d, d, ff))]
        lg, y, wts = _tensor(s.logits), _tensor(s.y[0]), _tensor(s.y[2])
        ids = _tensor(s.y[1])
        ids.type = B.I32

        def calls():
            c.graph_begin()
            c.moe_ffn(w[0], w[1], w[2], xs[0], lg, case["used"], CMIN, CMAX, y, ids, wts)
    else:
        prods = _products(case) if case["kind"] == "layer" else [(case["type"], case["m"], case["k"], 0)]
        s.y = [torch.empty(n, m, device="cuda") for _, m, _, _ in prods]
        todo = [(B.Tensor.weights(TYPES[t], w.data_ptr(), k, m), xs[i], _tensor(y)) for (t, m, k, i), w, y in zip(prods, s.w, s.y)]

        def calls():
            c.graph_begin()
            for w, x, y in todo:
                c.mul_mat(w, x, y)
    s.calls = calls
    if case["kind"] == "layer" or (case["kind"] == "moe" and n <= 8):
        torch.cuda.synchronize()
        calls()                                              # scratch grows outside the recording
        c.sync()
        s.graph = c.capture(calls)
        weakref.finalize(s, c.graph_free, s.graph)
    torch.cuda.synchronize()
    return s


def run(s):
    if s.graph is not None:
        _ctx().graph_launch(s.graph)
    else:
        s.calls()
    return s.y


def work(case):
    n = case["n"]
    if case["kind"] == "moe":
        pairs, e, d, ff = n * case["used"], case["experts"], case["d"], case["ff"]
        t = TYPES[case["type"]]
        one = 2 * ff * B.row_bytes(t, d) + d * B.row_bytes(t, ff)
        return {"bytes": min(pairs, e) * one + 4 * (2 * n * d + n * e + 2 * pairs), "flops": 2 * pairs * 3 * d * ff}
    prods = _products(case) if case["kind"] == "layer" else [(case["type"], case["m"], case["k"], 0)]
    xs = {i: k for _, _, k, i in prods}
    return {"bytes": sum(m * B.row_bytes(TYPES[t], k) + 4 * m * n for t, m, k, _ in prods) + sum(4 * n * k for k in xs.values()),
            "flops": sum(2 * m * k * n for _, m, k, _ in prods)}


def tolerance(case):
    # products: exact integer block dots, 32-bit float sums over the blocks of a row in any order; the MoE block rounds
    # its intermediate to 8 bits, where a last-bit difference moves a code by one now and then
    if case["kind"] == "moe":
        return {"rel": 2e-4, "max": 2e-2, "differ": 1e-4}
    return {"rel": 2e-6, "max": 2e-5}


def exact(case, seed):
    s = _inputs(case, seed)
    if case["kind"] != "moe":
        prods = _products(case) if case["kind"] == "layer" else [(case["type"], case["m"], case["k"], 0)]
        out = []
        for (t, m, k, i), w in zip(prods, s.w):
            x = _activation(t, s.x[i])
            out.append(torch.cat([x @ _dequantize(t, w[r:r + 4096], k).T for r in range(0, m, 4096)], -1))
        return out
    n, t, d, ff, e, used = case["n"], case["type"], case["d"], case["ff"], case["experts"], case["used"]
    p = torch.softmax(s.logits.double(), -1)
    top, ids = torch.topk(p, used, -1)
    wts = top / top.sum(-1, keepdim=True).clamp(CMIN, CMAX)
    x, y = _activation(t, s.x[0]), torch.zeros(n, d, dtype=torch.float64, device="cuda")
    wg, wu, wd = (w.view(e, m, -1) for w, m in zip(s.w, (ff, ff, d)))
    for q in torch.unique(ids).tolist():
        tok, slot = torch.nonzero(ids == q, as_tuple=True)
        a, b = x[tok] @ _dequantize(t, wg[q], d).T, x[tok] @ _dequantize(t, wu[q], d).T
        h = _activation(t, (a / (1 + torch.exp(-a)) * b).float())
        y.index_add_(0, tok, (h @ _dequantize(t, wd[q], ff).T) * wts[tok, slot][:, None])
    return [y, ids.to(torch.int32), wts]

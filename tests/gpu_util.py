"""Helpers shared by the GPU parity tests."""
import numpy as np

import arcint_b200 as A
import oracle as O


def rel_err(got, ref):
    """max relative error against max(|ref|, 1e-2 * max|ref| of the column)"""
    ref = np.asarray(ref, dtype=np.float64)
    floor = 1e-2 * np.abs(ref).max(axis=-1, keepdims=True)
    floor = np.maximum(floor, 1e-30)
    return float((np.abs(got - ref) / np.maximum(np.abs(ref), floor)).max())


def nmse(got, ref):
    ref = np.asarray(ref, dtype=np.float64)
    return float(((got - ref) ** 2).sum() / max((ref ** 2).sum(), 1e-300))


TOL = 1e-3          # max relative error against the fp64 product of the same quantized operands


def make_weights(t, m, k, seed, standin=True):
    """N(0, 0.02) weights quantized to type t (ggml rule for Q4_0/Q8_0, stand-in for the rest)."""
    return O.quantize(t, O.fill_normal(m * k, seed, 0.02).reshape(m, k))


def check_sums(got, t, w, k, x):
    """got against the fp64 product of the same quantized operands. The bound: block dots are exact integers and what is left are f32 sums over the K / 256 super-blocks (K / 32 blocks) of a
    row, each of at most three roundings of half an ulp (2^-24) of the running sum, so |error| <= 3 n 2^-24 sum|terms|; the sum of the
    absolute terms is taken from the operands."""
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


def normal_data(t, m, k, n, seed):
    """(packed N(0, 0.02) weights [m, .], N(0, 1) activations [n, k])"""
    rng = np.random.default_rng(seed)
    return O.quantize(t, O.fill_normal(m * k, seed, 0.02).reshape(m, k)), rng.normal(0, 1, size=(n, k)).astype(np.float32)

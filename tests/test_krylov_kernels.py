"""Single kernels of the linear solver (csrc/afx_implicit.cu) on crafted data."""
import ctypes

import numpy as np
import pytest

from tests import cuda

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hk(afx, tmp_path_factory):
    return cuda.load("krylov_harness", tmp_path_factory.mktemp("hk"), "afx_implicit.cu")


def _p(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _sq(hk, w, blocks):
    out = np.zeros(1)
    fn = hk.hk_sq_f32 if w.dtype == np.float32 else hk.hk_sq_f64
    assert fn(w.size, blocks, _p(w), _p(out)) == 0
    return out[0]


@pytest.mark.parametrize("scale", [2.0 ** 63, 2.0 ** 20, 1.0, 2.0 ** -20, 2.0 ** -40])
@pytest.mark.parametrize("lanes", [(0, 1, 2), (0, 7, 20), (5, 19, 31), (30, 17, 16)])
def test_fp32_sums_of_a_warp_hold_a_double_s_bits(hk, scale, lanes):
    """Three threads of a warp hold 1, 2^-25 and 2^-50 times the square of the
    scale: 51 bits, exact in FP64 in any order.  At 2^63 twelve more hold the
    largest, and the sum is beyond FP32's range."""
    w = np.zeros((256, 4), np.float32)  # a thread's 16-byte chunks
    if scale > 2.0 ** 60:
        w[3:15, 0] = scale
        w[lanes[0], 0] = scale
        w[lanes[2], 0] = scale * 2.0 ** -20
    else:
        w[lanes[0], 0] = scale
        w[lanes[1], :2] = scale * 2.0 ** -13  # two equal squares
        w[lanes[2], 0] = scale * 2.0 ** -25
    exact = float((np.sort(w.ravel()).astype(np.float64) ** 2).sum())
    assert _sq(hk, w.ravel(), 1) == exact


@pytest.mark.parametrize("n, blocks", [(4, 1), (4 * 250, 1), (4 * 257, 2), (4 * 5000, 20), (4 * 40000, 304)])
def test_norms_against_64_bits(hk, n, blocks):
    """FP64: some thirty additions of positive numbers, one rounding each.  FP32:
    integers of ten bits, so that a chunk's four squares are exact (22 bits) and
    the sum over the chunks, one per thread, has to be."""
    rng = np.random.default_rng(n)
    w = rng.standard_normal(n)
    assert abs(_sq(hk, w, blocks) - w @ w) <= 1e-14 * (w @ w)
    f = np.trunc(np.clip(w, -4.0, 4.0) * 2 ** 7).astype(np.float32)
    assert _sq(hk, f, blocks) == float((f.astype(np.float64) ** 2).sum())


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("k", [0, 3, 15, 16, 29])
@pytest.mark.parametrize("cells, blocks", [(60, 1), (3000, 12), (3000, 5)])
@pytest.mark.parametrize("near", [False, True])
def test_norm_of_the_new_vector_near_a_breakdown(hk, dtype, k, cells, blocks, near):
    """A product that lies in the span of the basis but for delta p (near): the
    first Gram-Schmidt pass leaves 1e-3 of it and the second has to find delta.
    The vector after the second pass is formed with a rounding per term, so its
    norm is good to (k + 3) units of the first remainder's; and since the last
    component is zero, the step gains nothing and the solve must not end."""
    rng = np.random.default_rng(cells + k)
    n, u = 4 * cells, float(np.finfo(dtype).eps)
    Q = np.linalg.qr(rng.standard_normal((n, k + 2)))[0]
    V = np.ascontiguousarray(Q[:, : k + 1].T.astype(dtype))
    c = rng.standard_normal(k + 1)
    c[k] = 0.0
    delta = u if near else 0.3
    w = (Q[:, : k + 1] @ c + delta * Q[:, k + 1]).astype(dtype)
    h1 = c * 1.001 if near else V.astype(np.float64) @ w.astype(np.float64)
    w0 = w.astype(np.float64)
    h2, st = np.zeros(k + 1), np.zeros(4)
    fn = hk.hk_cgs_f32 if dtype == np.float32 else hk.hk_cgs_f64
    w1 = w.copy()
    assert fn(n, k, blocks, _p(V), _p(w1), _p(h1), ctypes.c_double(1.0), ctypes.c_double(1e-2), _p(h2), _p(st)) == 0
    first = w1.astype(np.float64)  # after the first pass, as the kernel left it
    assert np.abs(first - (w0 - h1 @ V.astype(np.float64))).max() <= 2 * (k + 3) * u * np.abs(h1).max(initial=1.0)
    ref = np.linalg.norm(first - h2 @ V.astype(np.float64))
    assert abs(st[0] - ref) <= (k + 3) * u * np.linalg.norm(first)
    assert st[3] == k + 1
    if near and ref > 0.0:
        assert st[1] > 0.5 and st[2] == (1.0 if k == 29 else 0.0)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("threads", [1, 4])
@pytest.mark.parametrize("fwd", [0, 1])
@pytest.mark.parametrize("n", [1, 31, 129, 45000])
def test_one_colour_of_the_sweep(hk, dtype, threads, fwd, n):
    """x_p = D_p^-1 (r_p - sum O x_q) over one colour's rows, with one thread per
    row (colours of 40,000 rows and more) and with four, against 64 bits: up to
    sixteen products and a 4 x 4 block, forty roundings of terms of at most 4 + 16."""
    rng = np.random.default_rng(n + fwd)
    lo = max(n // 3, 8)  # rows of lower and of higher colours beside the colour's own
    N, c0 = n + 2 * lo, lo
    other = np.concatenate([np.arange(c0), np.arange(c0 + n, N)])
    col = np.where(rng.random((N, 4)) < 0.2, -1, rng.choice(other, (N, 4))).astype(np.int32)
    dinv, off = rng.uniform(-1, 1, (N, 4, 4)).astype(dtype), rng.uniform(-1, 1, (N, 4, 4, 4)).astype(dtype)
    r, x0 = rng.uniform(-1, 1, (N, 4)).astype(dtype), rng.uniform(-1, 1, (N, 4)).astype(dtype)
    # interleaved: 16-byte chunk c of slot s of row p is chunk (s * chunks + c) * N + p
    w = 16 // np.dtype(dtype).itemsize
    packed = np.ascontiguousarray(off.reshape(N, 4, 16 // w, w).transpose(1, 2, 0, 3))
    x = x0.copy()
    fn = hk.hk_gs_f32 if dtype == np.float32 else hk.hk_gs_f64
    assert fn(threads, N, c0, n, fwd, _p(col), _p(dinv), _p(packed), _p(r), _p(x)) == 0
    use = (col >= 0) & ((col < c0) if fwd else True)
    xo = np.where(use[..., None], x0[col].astype(np.float64), 0.0)
    s = r - np.einsum("pkij,pkj->pi", off.astype(np.float64), xo)
    ref = x0.astype(np.float64)
    ref[c0 : c0 + n] = np.einsum("pij,pj->pi", dinv.astype(np.float64), s)[c0 : c0 + n]
    assert np.abs(x - ref).max() <= 40 * np.finfo(dtype).eps * 20 * 4
    np.testing.assert_array_equal(np.delete(x, np.s_[c0 : c0 + n], 0), np.delete(x0, np.s_[c0 : c0 + n], 0))

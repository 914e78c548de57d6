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

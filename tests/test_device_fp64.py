"""On the GPU: the integer FP64 operations (csrc/afx_fp64.cuh) against the
device's own, bit for bit, on edge and random patterns; their reciprocal seeds
over every argument; and the face fluxes reversed by hand (csrc/afx_adjoint.cu)
against forward dual numbers through the flux itself."""
import ctypes

import numpy as np
import pytest

from tests import cuda

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ha(afx, tmp_path_factory):
    return cuda.load("adjoint_harness", tmp_path_factory.mktemp("ha"), "afx_adjoint.cu")


def _p(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _patterns(seed, n):
    """Every pair of edge values, then random signs, exponents (all of them, or
    the middle) and significands (random, few leading bits, ones at the end, the
    ends of a binade)."""
    edge = np.array([0.0, -0.0, 1.0, -1.0, 1.5, np.inf, -np.inf, np.nan, 5e-324, -2.5e-308, 2.2250738585072014e-308,
                     1.7976931348623157e308, float.fromhex("0x1.fffffffffffffp-1"),
                     float.fromhex("0x1.0000000000001p0"), 4.0, float.fromhex("0x1.fffffffffffffp0"), 1e-38, 1e-45,
                     3.4028235677973366e38, 3.4028234663852886e38, 1.17549435e-38, 1.1754943e-38])
    r = np.random.default_rng(seed)
    f = r.integers(0, 64, n)
    m = r.integers(0, 1 << 52, n, dtype=np.uint64)
    ones = (np.uint64(1) << r.integers(0, 52, n, dtype=np.uint64)) - np.uint64(1)
    m = np.where((f & 3) == 1, m & ~ones, np.where((f & 3) == 2, m | ones, m))
    end = r.integers(0, 4, n, dtype=np.uint64)
    m = np.where((f & 12) == 12, np.where(f & 16, np.uint64(0xFFFFFFFFFFFFF) - end, end), m)
    e = np.where(f & 32, r.integers(0, 2048, n), r.integers(850, 1200, n)).astype(np.uint64)
    x = (r.integers(0, 2, n, dtype=np.uint64) << np.uint64(63) | e << np.uint64(52) | m).view(np.float64)
    a, b = np.meshgrid(edge, edge)
    y = np.roll(x, 1)
    return np.concatenate([a.ravel(), x]), np.concatenate([b.ravel(), y])


@pytest.mark.parametrize("op", range(9))
def test_integer_operations_have_the_device_s_bits(ha, op):
    x, y = _patterns(op, 1 << 21)
    mine, theirs = np.zeros_like(x), np.zeros_like(x)
    assert ha.ha_ops(op, x.size, _p(x), _p(y), _p(mine), _p(theirs)) == 0
    same = (mine.view(np.uint64) == theirs.view(np.uint64)) | (np.isnan(mine) & np.isnan(theirs))
    if op == 8:
        same |= np.isnan(x)
    assert same.all(), (x[~same][:4], y[~same][:4], mine[~same][:4], theirs[~same][:4])


@pytest.mark.parametrize("root", [0, 1])
def test_seeds_stay_within_three_units(ha, root):
    """The operations allow the seeds three units in the last place (2^-24) either
    way; two is what the reciprocal's specification gives."""
    worst = np.zeros(2, np.int32)
    assert ha.ha_seeds(root, _p(worst)) == 0
    assert worst.max() <= 3 * 256, worst / 256.0


@pytest.mark.parametrize("visc", [0, 1])
@pytest.mark.parametrize("speed", ["below", "around", "above"])
def test_reversed_face_flux_is_the_forward_derivative(ha, visc, speed):
    """Eight (laminar: sixteen) directions per face.  `speed` puts the normal
    velocity on either side of the entropy fix's switch (5% of the speed of
    sound) and through the sonic point.  Tolerance: some four hundred roundings,
    amplified by at most 1 / (M^2 (gamma - 1)) < 250 where the pressure is the
    difference of the energies."""
    n, r = 4096, np.random.default_rng(17 + visc)
    ang = r.uniform(0, 2 * np.pi, n)
    nx, ny = np.cos(ang), np.sin(ang)
    lo, hi = {"below": (0.0, 0.04), "around": (0.03, 0.07), "above": (0.1, 1.3)}[speed]
    vn, vt = r.uniform(lo, hi, n) * r.choice([-1, 1], n), r.uniform(0.1, 0.6, n)

    def state():
        rho, p = 1.4 * (1 + 0.1 * r.standard_normal(n)).clip(0.5), (1 + 0.1 * r.standard_normal(n)).clip(0.5)
        u, v = vn * nx - vt * ny + 0.01 * r.standard_normal(n), vn * ny + vt * nx + 0.01 * r.standard_normal(n)
        return np.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)], 1)

    a = np.ascontiguousarray(np.concatenate([nx[:, None], ny[:, None], state(), state(), r.standard_normal((n, 12))], 1))
    mine, theirs = np.zeros((n, 16)), np.zeros((n, 16))
    args = [ctypes.c_double(v) for v in (1.4, 1 / 1.4, 0.05, 0.2)]
    assert ha.ha_face(visc, n, *args, _p(a), _p(mine), _p(theirs)) == 0
    scale = np.abs(theirs[:, :8]).max(axis=1, keepdims=True)
    assert (np.abs(mine - theirs) <= 1e-11 * scale).all(), np.abs((mine - theirs) / scale).max(axis=0)
    assert not np.array_equal(theirs[:, :4], 0 * theirs[:, :4])

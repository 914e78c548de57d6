"""The Venkatakrishnan constant outside its usual range, FP64: residuals against
the oracle, bit for bit.  With a negative constant the limiter's denominator
can vanish, where no bound on an FP32 estimate holds."""
import numpy as np
import pytest

from tests.cases import DEG, channel_case, gpu_solver, oracle_solver

pytestmark = pytest.mark.gpu


def _squares(n):
    """n x n unit squares, far field all round."""
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    a = (i * (n + 1) + j).ravel()
    k = np.arange(n)
    bedges = np.concatenate([np.stack([k, k + 1], 1), np.stack([k, k + 1], 1) + n * (n + 1),
                             np.stack([k * (n + 1), (k + 1) * (n + 1)], 1),
                             np.stack([k * (n + 1), (k + 1) * (n + 1)], 1) + n])
    m = dict(x=np.repeat(np.arange(n + 1.0), n + 1), y=np.tile(np.arange(n + 1.0), n + 1),
             cells=np.stack([a, a + n + 1, a + n + 2, a + 1], 1).astype(np.int32), bedges=bedges.astype(np.int32),
             bpatch=np.zeros(4 * n, np.int32), names=["farfield"])
    return m, {"farfield": dict(type="farfield", T=1.0, mach=0.3, angle=20 * DEG, p=1.0)}


def _check(afx, orc, m, bcs, q, k):
    so = oracle_solver(orc, m, bcs, limiter_k=float(k))
    so.init()
    so.set_q(q)
    g = gpu_solver(afx, m, bcs, limiter_k=float(k))
    g.init()
    g.set_q(q)
    np.testing.assert_array_equal(g.residual(), so.residual(), err_msg=str(k))
    return so


@pytest.mark.parametrize("n", [24, 208])  # both sides of 40,000 cells
def test_negative_constant_where_the_denominator_vanishes(afx, orc, n):
    """A state that is alike in x and y but for 1e-7, so the right and the upper
    face of a cell have nearly equal values, and constants that cancel their
    denominator to 1e-9 ... 1e-6 of its terms in one cell each."""
    m, bcs = _squares(n)
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    rng = np.random.default_rng(3)
    so = oracle_solver(orc, m, bcs)
    so.init()
    q = np.array(so.q()).reshape(-1, 4)
    wave = 0.01 * np.sin(0.37 * (i + j)).ravel()[:, None] * np.array([1.0, 0.7, 0.5, 1.3])
    q = (q * (1.0 + wave + 1e-9 * rng.standard_normal(q.shape))).ravel()
    so.set_q(q)
    so.residual()
    gx, r = so.get("gx").reshape(-1, 4), q.reshape(n, n, 4)
    for t in range(60):
        a, b, v = int(rng.integers(2, n - 2)), int(rng.integers(2, n - 2)), int(rng.integers(4))
        nb = [r[a, b, v], r[a + 1, b, v], r[a - 1, b, v], r[a, b + 1, v], r[a, b - 1, v]]
        g = 0.5 * gx[a * n + b, v]
        D = max(nb) - nb[0] if g > 0 else nb[0] - min(nb)
        base = D * D + 2 * g * g + D * abs(g)
        K = base * (1.0 - 10.0 ** rng.uniform(-9, -6) * rng.choice([-1.0, 1.0]))
        _check(afx, orc, m, bcs, q, -np.cbrt(K))


@pytest.mark.parametrize("k", [-20.0, -1.0, -0.0, 0.0, 1e-6, 1e4])
def test_residual_bits_over_the_constant(afx, orc, k):
    m, bcs, _ = channel_case(48, 26)
    so = oracle_solver(orc, m, bcs)
    so.init()
    q = np.array(so.q())
    _check(afx, orc, m, bcs, q * (1.0 + 1e-2 * np.random.default_rng(5).standard_normal(q.size)), k)

"""The FP64 limiter looks for the face that holds the least value in FP32 and
evaluates in FP64 only the faces that can hold it.  Its result has to be the
least value over all faces bit for bit, also where FP32 cannot tell: states
whose limiter values nearly tie (uniform flow, noise at and below FP32
resolution and at the 1e-16 threshold), strong jumps, and scales at which FP32
underflows; residuals against the oracle, triangles and quadrilaterals."""
import numpy as np
import pytest

from tests.cases import channel_case, gpu_solver, omesh_case, oracle_solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("noise", [0.0, 3e-16, 1e-15, 1e-12, 1e-9, 1e-7, 1e-5, 1e-3, 0.1])
@pytest.mark.parametrize("mesh", ["triangles", "quads", "channel"])
def test_residual_bits_where_limiter_values_tie(afx, orc, mesh, noise):
    if mesh == "channel":
        m, bcs, _ = channel_case(24, 13)
    else:
        m, bcs = omesh_case(33, 17, split=mesh == "triangles")
    so = oracle_solver(orc, m, bcs)
    so.init()
    q = np.array(so.q())
    rng = np.random.default_rng(7)
    q = q * (1.0 + noise * rng.standard_normal(q.size))
    if noise == 1e-3:  # one variable constant, one linear in the cell number
        q[2::4] = 0.0
        q[1::4] = 0.4 + 1e-4 * np.arange(q.size // 4)
    so.set_q(q)
    g = gpu_solver(afx, m, bcs)
    g.init()
    g.set_q(q)
    assert np.array_equal(g.residual(), so.residual())
    so.iterate(3)
    g.iterate(3)
    assert np.array_equal(g.get_q(), so.q())

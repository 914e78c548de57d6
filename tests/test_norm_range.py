"""The FP32-mixed residual norm: a cell's square is FP32, every sum over cells is
FP64, so the sum of a block's squares may pass FP32's range."""
import numpy as np
import pytest

from tests.cases import channel_case, gpu_solver, oracle_solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant, block", [("tile", 256), ("tile", 64), ("tile", 32), ("face", 256), ("gather", 128)])
def test_block_of_squares_beyond_fp32_range(afx, orc, variant, block):
    m, bcs, _ = channel_case(48, 26)
    bcs = {k: dict(b, p=1e17) if "p" in b else b for k, b in bcs.items()}
    so = oracle_solver(orc, m, bcs, second_order=False)
    so.init()
    q = np.array(so.q())
    q = q * (1.0 + 0.05 * np.random.default_rng(2).standard_normal(q.size))
    so.set_q(q)
    sq = (so.residual().reshape(-1, 4) ** 2).sum(axis=1)
    assert sq.max() < 1e38 and 256 * sq.mean() > 5e38  # (of the first stage; the last stage's are alike)
    ref = so.iterate(1)[-1]
    g = gpu_solver(afx, m, bcs, "fp32-mixed", second_order=False, kernel_variant=variant, block_size=block)
    g.init()
    g.set_q(q)
    # residuals of a noisy state: a few FP32 roundings of the fluxes each
    assert abs(g.iterate(1) - ref) <= 1e-5 * ref

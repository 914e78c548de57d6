"""Kernels that give a cell or a row one thread or four, by size (40,000 cells;
40,000 rows per launch of the linear solver): results on both sides of the
line, on sizes that fill neither a warp nor a block."""
import numpy as np
import pytest

from tests.cases import channel_case, gpu_solver, omesh_case, oracle_solver, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx, ny", [(5, 3), (141, 141), (142, 141)])  # 30, 39,762 and 40,044 triangles
@pytest.mark.parametrize("opts", [dict(), dict(gradient="least-squares", limiter="michalak"),
                                  dict(viscosity="laminar", mu_L=1e-4), dict(viscosity="laminar", second_order=False)])
def test_gradient_and_limiter_bits_on_both_sides_of_the_line(afx, orc, nx, ny, opts):
    m, bcs, q = channel_case(nx, ny)
    so = oracle_solver(orc, m, bcs, **opts)
    so.init()
    so.set_q(q)
    g = gpu_solver(afx, m, bcs, **opts)
    g.init()
    g.set_q(q)
    assert np.array_equal(g.residual(), so.residual())
    so.iterate(1)
    g.iterate(1)
    assert np.array_equal(g.get_q(), so.q())
    # FP32-mixed: an iteration adds increments below one with FP32's 6e-8 in each of
    # their few dozen operations
    f = gpu_solver(afx, m, bcs, "fp32-mixed", **opts)
    f.init()
    f.set_q(q)
    f.iterate(1)
    assert rel_l2(f.get_q(), so.q()) < 2e-6


@pytest.mark.parametrize("ns, nr", [(33, 17), (301, 151)])  # 561 and 45,451 rows
def test_implicit_solution_on_both_sides_of_the_line(afx, ns, nr):
    """FP64 and FP32-mixed (other Krylov arithmetic, same right-hand side) end at
    the same solution: each converged to 1e-10 of its start, the two agree to a
    hundred times that."""
    m, bcs = omesh_case(ns, nr, mach=0.4, split=False)
    out = []
    for prec in ("fp64", "fp32-mixed"):
        g = gpu_solver(afx, m, bcs, prec, solver="implicit", second_order=False, cfl=40.0)
        g.init()
        it, err = g.run_solver(1e-10, 300)
        assert err <= 1e-10, (prec, it, err)
        out.append(g.get_q())
    assert rel_l2(out[1], out[0]) < 1e-8


@pytest.mark.parametrize("ns, nr", [(33, 17), (301, 151)])
@pytest.mark.parametrize("gradient", ["green-gauss", "least-squares"])
def test_deformed_mesh_reaches_the_fp32_slot_records(afx, ns, nr, gradient):
    """Moving the wall by 1e-2 renews the geometry that FP32-mixed keeps per cell
    slot: one iteration agrees with FP64's as on the mesh it was created on."""
    m, bcs = omesh_case(ns, nr, mach=0.4, split=False)
    out = []
    for prec in ("fp64", "fp32-mixed"):
        g = gpu_solver(afx, m, bcs, prec, gradient=gradient)
        g.init()
        q = np.array(g.get_q())
        g.set_q(q * (1.0 + 0.01 * np.random.default_rng(4).standard_normal(q.size)))
        g.deform_patch(np.full(len(g.patch_nodes("wall")[0]), 1e-2), "wall")
        g.iterate(1)
        out.append(g.get_q())
    assert rel_l2(out[1], out[0]) < 2e-6

"""Batches whose cases differ in size by orders of magnitude: a case's norm is
summed by a cluster of blocks, most of which have no cell of a small case."""
import numpy as np
import pytest

from tests.cases import DEG, channel_case, gpu_settings, gpu_solver, oracle_solver, rel_l2

pytestmark = pytest.mark.gpu


def _batch(afx, cases, precision, **st):
    return afx.Batch([afx.mesh.from_arrays(m) for m, _ in cases],
                     [gpu_settings(afx, bcs, precision, **dict(st)) for _, bcs in cases])


def _strip(n, mach, aoa):
    """A row of n unit quadrilaterals: far field at the ends, walls above and below."""
    x = np.repeat(np.arange(n + 1.0), 2)
    y = np.tile([0.0, 1.0], n + 1)
    i = 2 * np.arange(n)
    bedges = [(0, 1), (2 * n, 2 * n + 1)] + [(k + s, k + 2 + s) for s in (0, 1) for k in i]
    m = dict(x=x, y=y, cells=np.stack([i, i + 2, i + 3, i + 1], axis=1).astype(np.int32),
             bedges=np.array(bedges, np.int32), bpatch=np.array([0, 0] + [1] * (2 * n), np.int32),
             names=["farfield", "wall"])
    bcs = {"farfield": dict(type="farfield", T=1.0, mach=mach, angle=aoa * DEG, p=1.0),
           "wall": dict(type="slip-wall")}
    return m, bcs


def _uneven_cases():
    big, bcs, _ = channel_case(200, 150, mach=0.3)
    return [_strip(1, 0.4, 2.0), _strip(7, 0.3, 1.0), (big, bcs), channel_case(15, 10, mach=0.5)[:2]]


@pytest.mark.parametrize("precision", ["fp64", "fp32-mixed"])
def test_batch_norms_of_very_uneven_cases(afx, orc, precision):
    # a cluster of blocks sums each case's norm: cases of 1, 7 and 300 cells
    # (most blocks of their clusters have no cell) beside one of 60,000.  FP64
    # as on each case alone (sums in another order); FP32-mixed the norms to a
    # few FP32 roundings of a single solver's, which holds its squares in FP32 too.
    cases = _uneven_cases()
    rng = np.random.default_rng(8)
    b = _batch(afx, cases, precision, kernel_variant="tile", block_size=128)
    b.init()
    qs = [b.get_q(c) * (1 + 1e-2 * rng.standard_normal(4 * b.n_real[c])) for c in range(len(cases))]
    assert [q.size // 4 for q in qs] == [1, 7, 60000, 300]
    for rep in range(20):
        for c, q in enumerate(qs):
            b.set_q(c, q)
        norms = b.iterate(3)
        if rep == 0:
            first = norms
        np.testing.assert_array_equal(norms, first)
    for c, (m, bcs) in enumerate(cases):
        if precision == "fp64":
            so = oracle_solver(orc, m, bcs)
            so.init()
            so.set_q(qs[c])
            no = so.iterate(3)[-1]
            np.testing.assert_array_equal(b.get_q(c), so.q())
            assert abs(norms[c] - no) <= 1e-12 * no
        else:
            g = gpu_solver(afx, m, bcs, precision, kernel_variant="tile", block_size=128)
            g.init()
            g.set_q(qs[c])
            no = g.iterate(3)
            assert rel_l2(b.get_q(c), g.get_q()) < 1e-12
            assert abs(norms[c] - no) <= 1e-12 * no


def test_implicit_batch_of_very_uneven_cases_isolates_a_failed_one(afx):
    # the same sums behind the right-hand side's finite check: each case in turn
    # is the one that is not finite
    cases = [c for k, c in enumerate(_uneven_cases()) if k != 2] + [channel_case(60, 40, mach=0.3)[:2]]
    imp = dict(solver="implicit", start_cfl=5.0, slope_cfl=0.0, max_cfl=5.0, second_order=False)
    for bad in range(len(cases)):
        b = _batch(afx, cases, "fp64", **imp)
        b.init()
        q = b.get_q(bad)
        q[::4] = np.nan
        b.set_q(bad, q)
        it, err, st = b.run_solver(1e-3, 3)
        assert [int(s) == 4 for s in st] == [c == bad for c in range(len(cases))], (bad, st)
        for c in range(len(cases)):
            if c != bad:
                assert np.isfinite(b.get_q(c)).all()

"""Natural-order sweeps of small systems in one block on the GPU.

The block sweeps replace the sync-free ones where a system's vectors fit one block.  At the sizes around
the limit and at 1 to 16 systems the solves must reach the solutions of the oracle's own COCG13_single
(its true residual of the device solution at the asked tolerance), for FP64 and for the FP32 inner solve.
"""
import numpy as np
import pytest

from actfemtide_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fw(gpulib):
    from actfemtide_b200.forward import Forward
    f = Forward(0)
    yield f
    f.close()


# edges: 98, 878, 3,256 (16 systems: past the limit), 9,972 and 11,448 (either side of 10,240 rows of one system)
@pytest.mark.parametrize("dims,ns", [((2, 2, 2), 1), ((4, 4, 6), 1), ((4, 4, 6), 2), ((3, 4, 5), 8), ((2, 3, 4), 16),
                                     ((8, 8, 6), 4), ((8, 8, 6), 16), ((11, 11, 10), 1), ((12, 11, 11), 1)])
def test_ssor_solutions(fw, oracle, dims, ns):
    m = synth.tidal_box(*dims, seed=3, block=False, site_grid=(-5.0, 5.0), half_km=10.0)
    fw.load_model(m)
    fw.set_sigma(np.maximum(m.sigma_per_tet(), 1e-2))  # conductive enough for plain SSOR to converge quickly
    fw.assemble()
    of = oracle.OracleForward(m)
    A = oracle.forward_assemble(m, of.line, of.n6line, oracle.pattern(len(of.line), of.n6line), m.freqs[0],
                                np.maximum(m.sigma_per_tet(), 1e-2))
    for precision in ("fp64", "mixed"):
        tol = 1e-9 if precision == "fp64" else 1e-7
        r = fw.solve(np.full(ns, m.freqs[0]), precond="SSOR", precision=precision, tol=tol, maxit=20000)
        if precision == "fp64":
            assert r.ok, r
        for k in {0, ns - 1}:
            assert oracle.true_residual(A, fw.solution(k)) <= 1.01 * max(tol, r.resid_true)


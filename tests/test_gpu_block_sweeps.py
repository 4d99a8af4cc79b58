"""Natural-order sweeps (SSOR) on either side of the one-block limit (GPU).

Up to 160 KB of vector values (10,240 rows x systems in FP64, 20,480 in FP32) a sweep runs in one block, above
by bounded waits.  Both have to be the oracle's COCG13_single: its iterates after one and five iterations
(1e-9 of the largest entry, as for the tiny mesh), and a solve with the FP32 inner iteration has to converge to
1e-8 in the oracle's own residual.
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


def _system(fw, oracle, dims, sigma):
    m = synth.tidal_box(*dims, seed=3, block=False, site_grid=(-5.0, 5.0), half_km=10.0)
    fw.load_model(m)
    fw.set_sigma(sigma(m))
    fw.assemble()
    of = oracle.OracleForward(m)
    return m, oracle.forward_assemble(m, of.line, of.n6line, oracle.pattern(len(of.line), of.n6line), m.freqs[0], sigma(m))


# rows x systems: 878 and 7,024 (inside), 9,525 and 11,353 (either side in FP64), 14,048 (inside in FP32 only), 25,520
CASES = [((4, 4, 6), 1), ((4, 4, 6), 8), ((11, 11, 10), 1), ((12, 11, 11), 1), ((4, 4, 6), 16), ((8, 8, 6), 8)]


@pytest.mark.parametrize("dims,ns", CASES)
def test_iterates_are_the_oracles(fw, oracle, dims, ns):
    m, A = _system(fw, oracle, dims, lambda m: np.maximum(m.sigma_per_tet(), 1e-2))
    for its in (1, 5):
        r = fw.solve(np.full(ns, m.freqs[0]), precond="SSOR", tol=1e-30, maxit=its)
        assert r.iterations == its
        x = oracle.cocg13_single(A, precond="SSOR", resid=1e-30, maxit=its)["x"]
        for k in {0, ns - 1}:
            assert np.abs(fw.solution(k) - x).max() <= 1e-9 * np.abs(x).max()


@pytest.mark.parametrize("dims,ns", CASES)
def test_fp32_inner_solves_converge(fw, oracle, dims, ns):
    m, A = _system(fw, oracle, dims, lambda m: np.ones(m.ntet))
    r = fw.solve(np.full(ns, m.freqs[0]), precond="SSOR", precision="mixed", tol=1e-8, maxit=20000)
    assert r.ok and r.resid_true <= 1e-8, r
    for k in {0, ns - 1}:
        assert oracle.true_residual(A, fw.solution(k)) <= 1.01e-8

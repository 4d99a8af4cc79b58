"""Accuracy of the solution vector itself (AFEM_PRECOND_HYBRID), not of its residual.

On the gradients the system is i omega M alone, 1e-12 of the rest in the air: a residual at rounding level
still leaves the FP64 recursion's solution 1e-6 from the system's (1.2e-6 with the colour sweeps on this
mesh, 2.1e-6 with the polynomial smoother), whatever the tolerance.  The solver forms its residual anew once
in extended precision, after which the two halves of a solve hold 1e-6 times the other's reduction each;
the bound is 5e-7, below what any solve without that step leaves.  The reference solution is a sparse LU
refined by residuals in 80-bit arithmetic.
"""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as sla

from actfemtide_b200 import synth

pytestmark = pytest.mark.gpu
BOUND = 5e-7


@pytest.fixture(scope="module")
def fw(gpulib):
    from actfemtide_b200.forward import Forward
    f = Forward(0)
    yield f
    f.close()


def _model(seed):
    return synth.tidal_box(12, 12, 9, seed=seed, grf=True, block=False)


def _solution(e):
    """The exported system's solution to about 1e-15 of its norm."""
    n = len(e["D"])
    A = (sp.diags(e["D"]) + sp.csr_matrix((e["AU"], e["IAU"] - 1, e["INU"]), shape=(n, n))
         + sp.csr_matrix((e["AL"], e["IAL"] - 1, e["INL"]), shape=(n, n))).tocsr()
    lu = sla.splu(A.tocsc(), permc_spec="MMD_AT_PLUS_A", options=dict(SymmetricMode=True), diag_pivot_thresh=0.0)
    x = lu.solve(e["b"]).astype(np.clongdouble)
    data = A.data.astype(np.clongdouble)
    for _ in range(5):
        r = e["b"].astype(np.clongdouble) - np.add.reduceat(data * x[A.indices], A.indptr[:-1])
        d = lu.solve(r.astype(np.complex128))
        x = x + d
    assert np.linalg.norm(d) < 1e-8 * np.linalg.norm(x.astype(np.complex128))
    return x.astype(np.complex128)


def _off(x, ref):
    return np.linalg.norm(x - ref) / np.linalg.norm(ref)


@pytest.fixture(scope="module")
def system(fw):
    m = _model(1)
    fw.load_model(m)
    fw.assemble()
    return m, _solution(fw.export_system(m.freqs[0]))


@pytest.mark.parametrize("precision", ["fp64", "pc32"])
@pytest.mark.parametrize("ns,launches,check_every", [(1, False, 0), (4, False, 0), (16, False, 0), (1, True, 0),
                                                     (16, True, 0), (2, True, 6), (8, True, 0)])
def test_the_solution_itself(fw, system, precision, ns, launches, check_every):
    m, ref = system
    fw.load_model(m)
    fw.assemble()
    fw.set_profiling(launches)  # the launches of large systems, where the one-launch form would run
    r = fw.solve(np.full(ns, m.freqs[0]), precond="HYBRID", precision=precision, tol=1e-10, maxit=2000,
                 check_every=check_every)
    fw.set_profiling(False)
    assert r.ok, r
    assert max(_off(fw.solution(k), ref) for k in range(ns)) < BOUND


def test_the_solutions_of_a_packed_batch(fw):
    parts = [_model(1), synth.tidal_box(7, 8, 6, seed=3, grf=True, block=False), _model(2)]
    refs = []
    for m in parts:
        fw.load_model(m)
        fw.assemble()
        refs.append(_solution(fw.export_system(m.freqs[0])))
    fw.load_packed(synth.pack(parts))
    fw.assemble()
    r = fw.solve(np.array([m.freqs[0] for m in parts]), precond="HYBRID", tol=1e-10, maxit=2000)
    assert r.ok, r
    assert max(_off(fw.solution(k), x) for k, x in enumerate(refs)) < BOUND

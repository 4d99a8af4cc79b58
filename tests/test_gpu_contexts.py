"""Contexts beside one another and at their end on the GPU (afem_create, afem_destroy; one per host thread)."""
import numpy as np
import pytest

from actfemtide_b200 import capi, synth
from actfemtide_b200.capi import AfemError

pytestmark = pytest.mark.gpu


def test_context_closed_right_after_a_failed_call(gpulib):
    """Closing frees the context's memory only after its stream: the next context starts clean."""
    from actfemtide_b200.forward import Forward
    m = synth.small_model()
    with Forward(0) as keep:
        keep.load_model(m)
        keep.assemble()
        ref = keep.solve(m.freqs[0], precond="HYBRID", tol=1e-9)
        x = keep.solution(0)
        for _ in range(3):
            fw = Forward(0)
            fw.load_model(m)
            fw.assemble()
            b = np.zeros((fw.nline, 1), np.complex128)
            b[100], b[200] = 1.0, 1.0j  # b^T b = 0: rho vanishes in the first iteration
            with pytest.raises(AfemError) as e:
                fw.solve_rhs(m.freqs[0], b, precond="NONE", tol=1e-8, maxit=100)
            assert e.value.code == capi.STATUS_CODE["AFEM_EBREAKDOWN"]
            fw.close()
            again = keep.solve(m.freqs[0], precond="HYBRID", tol=1e-9)
            assert again.iterations == ref.iterations and np.array_equal(keep.solution(0), x)

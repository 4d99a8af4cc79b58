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


@pytest.mark.parametrize("precond", ["HYBRID", "SSOR"])
def test_two_threads_with_meshes_of_two_sizes(gpulib, precond):
    """A kernel's limit of shared memory belongs to the device: one context's mesh must not lower another's."""
    import threading

    from actfemtide_b200.forward import Forward
    models = [synth.tidal_box(*d, seed=4, block=False, half_km=10.0) for d in ((9, 9, 8), (4, 4, 4))]
    if precond == "SSOR":
        models = [synth.tidal_box(*d, seed=4, block=False, half_km=10.0) for d in ((7, 7, 6), (3, 3, 3))]
    errors, got = [], [[], []]

    def work(k):
        try:
            m = models[k]
            with Forward(0) as fw:
                fw.load_model(m)
                fw.set_sigma(np.maximum(m.sigma_per_tet(), 1e-2))
                fw.assemble()
                fw.set_profiling(precond == "HYBRID")  # every kernel launched by itself
                for _ in range(12):
                    r = fw.solve(m.freqs[0], precond=precond, tol=1e-8, maxit=400 if precond == "SSOR" else 2000,
                                 use_graph=False)
                    got[k].append((r.status, r.iterations, fw.solution(0)))
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for runs in got:
        assert len(runs) == 12
        for status, its, x in runs[1:]:
            assert (status, its) == runs[0][:2] and np.array_equal(x, runs[0][2])

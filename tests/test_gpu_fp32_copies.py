"""FP32 copies that a solve with the FP32 preconditioner makes (GPU): those that its iteration reads."""
import numpy as np
import pytest

from actfemtide_b200 import capi, synth

pytestmark = pytest.mark.gpu


def test_multicolour_sweeps_convert_their_own_rows_only(gpulib):
    """SSOR_MC reads the colour-ordered rows: two conversions an assembly (lower, upper), not a third one of the
    whole matrix.  Counted as launches of a capped solve beyond those of the FP64 preconditioner."""
    from actfemtide_b200.forward import Forward
    m = synth.tidal_box(6, 6, 5, seed=1, half_km=10.0)
    with Forward(0) as fw:
        fw.load_model(m)
        fw.set_spmv_rows_per_warp(1)  # no timing runs
        count = {}
        for precision in ("fp64", "pc32"):
            for _ in range(2):  # the second with buffers and tables at hand
                fw.assemble()
                before = capi.lib().afem_launch_count()
                fw.solve(np.full(1, m.freqs[0]), precond="SSOR_MC", precision=precision, tol=1e-10, maxit=8,
                         use_graph=False)
                count[precision] = capi.lib().afem_launch_count() - before
        assert count["pc32"] - count["fp64"] == 2


def test_nodal_sweeps_convert_their_own_rows_only(gpulib):
    """The nodal sweeps read the nodal matrix by its colour-ordered halves: four conversions an assembly (the edges'
    halves, the nodes' halves), not a fifth one of the nodal matrix in row order.  Counted as above."""
    from actfemtide_b200.forward import Forward
    m = synth.tidal_box(6, 6, 5, seed=1, half_km=10.0)
    with Forward(0) as fw:
        fw.load_model(m)
        fw.set_spmv_rows_per_warp(1)
        count = {}
        for precision in ("fp64", "pc32"):
            for _ in range(2):
                fw.assemble()
                before = capi.lib().afem_launch_count()
                fw.solve(np.full(1, m.freqs[0]), precond="HYBRID", precision=precision, tol=1e-10, maxit=8,
                         sigma_diag=1.5, use_graph=False)
                count[precision] = capi.lib().afem_launch_count() - before
        assert count["pc32"] - count["fp64"] == 4

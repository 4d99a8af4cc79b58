"""Network kernels at the edges of their tiles: gradients against the CPU reference.

A handful of 64-row tiles with a ragged last one, and enough tiles that a block of the backward kernel
takes more than one; there the residual lives on a few hundred rows (the first, the last, those where the
blocks' second tiles begin), so that no tile's part drowns in the others'.  Tolerances as for the other
network tests: BF16 weights and activations with FP32 accumulation against a reference with the same
roundings (loss 2e-2, gradient cosine 0.99, norm within 5 %).
"""
import numpy as np
import pytest

from actfemtide_b200 import learned, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,first,last", [((3, 3, 3), 0, None), ((4, 3, 3), 0, None), ((16, 16, 12), 0, 300),
                                              ((16, 16, 12), -300, None), ((16, 16, 12), 11700, 12000)])
def test_gradient_matches_cpu(gpulib, shape, first, last):
    from oracle import mpnn_ref as R
    from test_gpu_learned import ref_graph
    from actfemtide_b200.forward import Forward
    fw = Forward(0)
    m = synth.tidal_box(*shape, seed=3, site_grid=(-6.0, 0.0, 6.0), half_km=12.0)
    fw.load_model(m)
    fw.assemble()
    f = m.freqs[0]
    g = ref_graph(fw, m, f)
    rng = np.random.default_rng(0)
    p = learned.init_params(1)
    p[-2 * learned.H:] = rng.standard_normal(2 * learned.H) * 0.1
    P = learned.unflatten(p)
    fw.mpnn_set_params(p)
    r = rng.standard_normal(fw.nline) + 1j * rng.standard_normal(fw.nline)
    keep = np.zeros(fw.nline, bool)
    keep[first:last] = True
    r[~keep] = 0.0
    loss, grad = fw.mpnn_loss_grad(f, r[None, :])
    lref, G = R.grad(P, g, r, bf16=True)
    assert abs(loss - lref) <= 2e-2 * lref
    ref = learned.flatten(G).astype(np.float64)
    cos = float(grad @ ref / (np.linalg.norm(grad) * np.linalg.norm(ref)))
    assert cos >= 0.99, cos
    assert abs(np.linalg.norm(grad) / np.linalg.norm(ref) - 1.0) <= 0.05
    fw.close()

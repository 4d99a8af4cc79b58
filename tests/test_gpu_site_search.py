"""Element search of many sites in few tetrahedra (GPU): the sites are shared out in groups of 64 to 512.

Each site's element, columns and values must be those of a search of a few sites at a time, and the element
the one of lowest id that holds the site (barycentric coordinates in 64 bits).
"""
import numpy as np
import pytest

from actfemtide_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nobs", [1, 63, 64, 65, 513, 1025, 20000])
@pytest.mark.parametrize("dims", [(2, 2, 2), (6, 5, 4)])
def test_groups_of_sites(gpulib, dims, nobs):
    from actfemtide_b200.forward import Forward
    m = synth.tidal_box(*dims, block=False, half_km=10.0)
    rng = np.random.default_rng(nobs)
    pts = rng.uniform(-9.9, 9.9, (nobs, 3))
    with Forward(0) as fw:
        fw.load_model(m)
        item, ve, vf, iele = fw.site_coeffs(pts)
        some = rng.choice(nobs, min(nobs, 64), replace=False)
        for i in some:
            one = fw.site_coeffs(pts[i:i + 1])
            assert np.array_equal(item[i], one[0][0]) and iele[i] == one[3][0]
            assert np.array_equal(ve[:, i], one[1][:, 0]) and np.array_equal(vf[:, i], one[2][:, 0])
    p = m.xyz[m.n4 - 1]
    inv = np.linalg.inv(p[:, 1:] - p[:, :1])  # rows of (x - p0) inv: the coordinates 1..3
    for i in some:
        lam = np.einsum("tc,tcj->tj", pts[i] - p[:, 0], inv)
        low = np.minimum(lam.min(axis=1), 1 - lam.sum(axis=1))
        assert low[iele[i] - 1] > -1e-9 and not np.any(low[:iele[i] - 1] > 1e-9)

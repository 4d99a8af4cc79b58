"""Coarse correction of the gradient-corrected COCG on the GPU (AFEM_PRECOND_HYBRID).

The solution must be the system's own: the oracle's FP64 true residual of the device solution at the
asked tolerance, and (small meshes) site fields within 1e-6 of a direct solve of the oracle's assembly.
The meshes are where the grids and the cycle can go wrong: two planes on an axis, odd and even plane
counts, one flat axis, graded cells, jittered nodes (every node inside a cell), a mesh below the
correction's minimum, level-1 grids on both sides of the one-block cycle's limit, packed batches.
"""
import dataclasses

import numpy as np
import pytest
import scipy.sparse.linalg as sla

from actfemtide_b200 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fw(gpulib):
    from actfemtide_b200.forward import Forward
    f = Forward(0)
    yield f
    f.close()


def _jitter(m, amp):
    """The mesh with its interior nodes moved by up to amp of the smallest cell (tags and orientation kept)."""
    rng = np.random.default_rng(5)
    lo, hi = m.xyz.min(axis=0), m.xyz.max(axis=0)
    h = (hi - lo) / m.dims
    inner = np.all((m.xyz > lo + 0.5 * h) & (m.xyz < hi - 0.5 * h), axis=1)
    xyz = m.xyz + inner[:, None] * rng.uniform(-amp, amp, m.xyz.shape) * h
    sites = m.sites + np.array([0.3, 0.2, -0.4])
    return dataclasses.replace(m, xyz=xyz, sites=sites)


CASES = {
    "2x2x4_below_minimum": lambda: synth.tiny_model(),
    "3x5x4": lambda: synth.tidal_box(3, 5, 4, seed=1, block=False, site_grid=(-5.0, 5.0), half_km=10.0),
    "12x2x6_flat": lambda: synth.tidal_box(12, 2, 6, seed=2, grf=True, block=False),
    "9x10x7": lambda: synth.tidal_box(9, 10, 7, seed=3, grf=True, block=False),
    "8x8x8_jittered": lambda: _jitter(synth.tidal_box(8, 8, 8, seed=4, grf=True, block=False), 0.2),
}


@pytest.mark.parametrize("precision", ["fp64", "pc32"])
@pytest.mark.parametrize("name", CASES)
def test_small_meshes_match_a_direct_solve(fw, oracle, name, precision):
    m = CASES[name]()
    of = oracle.OracleForward(m)
    A = of.assemble(m.freqs[0])
    x = sla.spsolve(A.to_scipy().tocsc(), A.b)
    ref = np.asarray(of.sites(x, m.freqs[0])[0]).reshape(5, -1)
    fw.load_model(m)
    fw.assemble()
    for ns in (1, 2, 16):
        r = fw.solve(np.full(ns, m.freqs[0]), precond="HYBRID", precision=precision, tol=1e-9, maxit=2000)
        assert r.ok and r.resid_true <= 1e-9, (ns, r)
        assert oracle.true_residual(A, fw.solution(ns - 1)) <= 1.01e-9
        out = fw.sites(m.sites)
        assert np.abs(out - ref).max() <= 1e-6 * np.abs(ref).max()


@pytest.mark.parametrize("dims", [(22, 22, 22), (24, 24, 20), (40, 26, 17)])
def test_grids_around_the_one_block_limit(fw, oracle, dims):
    """Level-1 grids of 12^3 = 1,728, 13 x 13 x 11 = 1,859 and about 21 x 14 x 9 nodes: launches for the first
    level, one block below; the iteration count stays that of a mesh a quarter as wide."""
    m = synth.tidal_box(*dims, seed=6, grf=True, block=False)
    of = oracle.OracleForward(m)
    A = of.assemble(m.freqs[0])
    fw.load_model(m)
    fw.assemble()
    for ns, precision in ((1, "fp64"), (4, "pc32"), (8, "fp64")):
        r = fw.solve(np.full(ns, m.freqs[0]), precond="HYBRID", precision=precision, tol=1e-9, maxit=2000)
        assert r.ok and r.iterations < 90, (ns, r)
        assert oracle.true_residual(A, fw.solution(ns - 1)) <= 1.01e-9


def test_mixed_precision_uses_the_correction(fw):
    """FP32 inner solve (conductive everywhere, where FP32 holds): converges with the correction in FP32."""
    m = synth.tidal_box(10, 9, 8, seed=7, block=False)
    fw.load_model(m)
    fw.set_sigma(np.ones(m.ntet))
    fw.assemble()
    r = fw.solve([m.freqs[0]] * 2, precond="HYBRID", precision="mixed", tol=1e-8, maxit=5000)
    assert r.ok and r.resid_true <= 1e-8, r


@pytest.mark.parametrize("precision", ["fp64", "pc32"])
def test_packed_meshes_of_different_depth(fw, oracle, precision):
    """Packed meshes whose hierarchies have different numbers of levels, one of them a handful of cells."""
    parts = [synth.tidal_box(nx, ny, nz, seed=20 + k, field_seed=30 + k, grf=True, block=False, name=f"p{k}")
             for k, (nx, ny, nz) in enumerate([(2, 3, 2), (9, 8, 7), (20, 6, 11), (26, 25, 20)])]
    pk = synth.pack(parts)
    fw.load_packed(pk)
    fw.assemble()
    r = fw.solve([m.freqs[0] for m in parts], precond="HYBRID", precision=precision, tol=1e-9, maxit=3000)
    assert r.ok, r
    for k, m in enumerate(parts):
        A = oracle.OracleForward(m).assemble(m.freqs[0])
        assert oracle.true_residual(A, fw.solution(k)) <= 1.01e-9


def test_new_conductivities_and_bounds_rebuild_the_matrices(fw, oracle):
    """The Galerkin matrices follow the assembly: other conductivities, then other Dirichlet bounds."""
    m = synth.tidal_box(8, 9, 8, seed=9, grf=True, block=False)
    fw.load_model(m)
    for sig, dz in ((m.sigma_land, 0.0), (m.sigma_land[::-1].copy(), 0.0), (m.sigma_land, 13.0)):
        m2 = dataclasses.replace(m, sigma_land=sig, bounds=dict(m.bounds, zmax=m.bounds["zmax"] - dz))
        fw.set_cond(m2.sigma_air, m2.sigma_ocean, 1, sigma_file=m2.sigma_land)
        b = m2.bounds
        fw.set_bounds(b["zmin"], b["zmax"], b["xout"], b["yout"])
        fw.assemble()
        A = oracle.OracleForward(m2).assemble(m2.freqs[0])
        r = fw.solve(m2.freqs[0], precond="HYBRID", tol=1e-9, maxit=2000)
        assert r.ok and oracle.true_residual(A, fw.solution(0)) <= 1.01e-9, r


@pytest.mark.parametrize("ns", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("precision", ["fp64", "pc32"])
def test_one_launch_iteration_gives_the_same_solution(fw, oracle, ns, precision):
    """Small systems iterate inside one launch, profiled solves by a launch per step: the same polynomial,
    cycles and formulas, so both reach the tolerance and their site fields agree to 1e-6.  The caps on
    iterations and an iteration count that ends inside a launch hold for both."""
    m = synth.tidal_box(9, 8, 10, seed=12, grf=True, block=False)
    fw.load_model(m, sources=[(m.F, m.v), (m.F, 0.5j * m.v)])
    fw.assemble()
    f = 1.0 / (3600.0 * np.array((synth.BATCH_PERIODS_H * 2)[:ns]))
    src = np.arange(ns) % 2
    kw = dict(precond="HYBRID", precision=precision)
    r = fw.solve(f, src, tol=1e-9, maxit=2000, **kw)
    assert r.ok and r.resid_true <= 1e-9, r
    one = fw.sites(m.sites)
    A = oracle.OracleForward(m).assemble(f[0])
    assert oracle.true_residual(A, fw.solution(0)) <= 1.01e-9
    fw.set_profiling(True)  # launches per step
    r2 = fw.solve(f, src, tol=1e-9, maxit=2000, **kw)
    fw.set_profiling(False)
    assert r2.ok and abs(r2.iterations - r.iterations) <= 3, (r, r2)
    assert np.abs(fw.sites(m.sites) - one).max() <= 1e-6 * np.abs(one).max()
    for cap in (1, 7):  # EMAXITER with exactly that many iterations
        rc = fw.solve(f, src, tol=1e-9, maxit=cap, **kw)
        assert rc.status == -4 and rc.iterations == cap, rc
    rc = fw.solve(f, src, tol=1e-9, maxit=2000, check_every=5, **kw)
    assert rc.ok and rc.iterations == r.iterations


def test_packed_iterates_do_not_depend_on_the_companions(fw):
    """The smoother's interval is each mesh's own: after 12 iterations a mesh's iterate is the same, but for
    the order of sums (1e-16 a step, grown at most a thousandfold each by the iteration's scalars), whatever
    it is packed with."""
    a = synth.tidal_box(7, 8, 6, seed=3, grf=True, block=False)
    others = [synth.tidal_box(8, 8, 6, seed=2, block=False), synth.tidal_box(20, 3, 9, seed=2, grf=True, block=False)]
    xs = []
    for b in others:
        fw.load_packed(synth.pack([a, b]))
        fw.assemble()
        r = fw.solve(np.full(2, a.freqs[0]), precond="HYBRID", tol=1e-12, maxit=12)
        assert r.iterations == 12
        xs.append(fw.solution(0))
    assert np.linalg.norm(xs[0] - xs[1]) < 1e-9 * np.linalg.norm(xs[0])


def test_thin_elements_do_not_break_the_smoother(fw):
    """Ten nodes moved to 1/200 of their way from a face of one of their tetrahedra: the smoother stays positive
    on the eigenvalues these add, and they may cost half as many iterations again, not twice as many."""
    m = synth.tidal_box(16, 16, 12, seed=4, grf=True, block=False)
    rng = np.random.default_rng(3)
    xyz = m.xyz.copy()
    lo, hi = xyz.min(axis=0), xyz.max(axis=0)
    h = (hi - lo) / m.dims
    sign = np.sign(_volumes(xyz, m.n4))
    inner = np.where(np.all((xyz > lo + 1.5 * h) & (xyz < hi - 1.5 * h), axis=1))[0]
    used, moved = set(), 0
    for a in rng.permutation(inner):
        around = np.where((m.n4 == a + 1).any(axis=1))[0]
        nodes = set((m.n4[around] - 1).ravel())
        if used & nodes:
            continue
        face = [b for b in m.n4[around[rng.integers(len(around))]] - 1 if b != a]
        old = xyz[a].copy()
        xyz[a] = 0.005 * old + 0.995 * xyz[face].mean(axis=0)
        if np.all(_volumes(xyz, m.n4[around]) * sign[around] > 0):
            used |= nodes
            moved += 1
            if moved == 10:
                break
        else:
            xyz[a] = old
    assert moved == 10
    its = []
    for q in (m, dataclasses.replace(m, xyz=xyz)):
        fw.load_model(q)
        fw.assemble()
        r = fw.solve(q.freqs[0], precond="HYBRID", tol=1e-9, maxit=2000)
        assert r.ok, r
        its.append(r.iterations)
    assert its[1] <= 1.5 * its[0], its


def _volumes(xyz, n4):
    p = xyz[n4 - 1]
    return np.linalg.det(p[:, 1:] - p[:, :1]) / 6


def _refined_around(points, count, n=10, half=50.0):
    """A Delaunay mesh of a jittered n^3 grid with `count` more nodes around each point, 20 m to 4 km from it."""
    from scipy.spatial import Delaunay
    rng = np.random.default_rng(0)
    g = np.stack(np.meshgrid(*[np.linspace(-half, half, n + 1)] * 3, indexing="ij"), -1).reshape(-1, 3)
    g += np.all(np.abs(g) < half - 1e-6, axis=1)[:, None] * rng.uniform(-0.5, 0.5, g.shape) * half / n
    xyz = [g]
    for p in points:
        d = rng.normal(size=(count, 3))
        xyz.append(p + d / np.linalg.norm(d, axis=1)[:, None] * np.exp(rng.uniform(np.log(0.02), np.log(4.0), (count, 1))))
    xyz = np.concatenate(xyz)
    n4 = Delaunay(xyz, qhull_options="QJ Pp").simplices + 1
    like = synth.tidal_box(2, 2, 2, block=False)
    vol, sign = _volumes(xyz, n4), np.sign(_volumes(like.xyz, like.n4)[0])
    q = xyz[n4 - 1]
    edge = np.abs(q[:, [0, 0, 0, 1, 1, 2]] - q[:, [1, 2, 3, 2, 3, 3]]).max(axis=(1, 2))
    keep = np.abs(vol) > 1e-9 * edge ** 3  # (flat ones on the box's faces)
    n4 = np.where((np.sign(vol) != sign)[:, None], n4[:, [0, 2, 1, 3]], n4)[keep]
    cen = xyz[n4 - 1].mean(axis=1)
    tag = np.where(cen[:, 2] > 0, 1, np.where((cen[:, 2] > -5) & (cen[:, 0] < 0), 2, 3)).astype(np.int32)
    order = np.argsort(tag, kind="stable")
    n4, tag = n4[order], tag[order]
    sea = np.zeros(len(xyz), bool)
    sea[n4[tag == 2] - 1] = True
    perm = np.argsort(~sea, kind="stable")
    new = np.empty(len(xyz), np.int64)
    new[perm] = np.arange(len(xyz))
    nodes = int(sea.sum())
    return dataclasses.replace(like, xyz=np.ascontiguousarray(xyz[perm]), n4=(new[n4 - 1] + 1).astype(np.int32), tag=tag,
                               sigma_land=np.full(int((tag == 3).sum()), 0.01), nodes=nodes,
                               F=np.tile(np.array(synth.F_MAIN_NT), (nodes, 1)), v=np.full((nodes, 3), 0.05 + 0.01j),
                               bounds=dict(zmin=-half, zmax=half, xout=half, yout=half))


@pytest.mark.parametrize("count,smoothed", [(100, True), (4000, False)])
def test_nodes_crowded_around_points_keep_the_sweeps(fw, count, smoothed):
    """Regions of fine elements around four points: with thousands of nodes in a cell of the tensor grid the
    solve takes the colour sweeps (their kernels in the profile); either way it converges."""
    m = _refined_around([(-35.0, -18.0, -3.0), (-12.0, 35.0, -12.0), (13.0, -36.0, -25.0), (34.0, 12.0, -38.0)], count)
    fw.load_model(m)
    fw.assemble()
    fw.set_profiling(True)
    r = fw.solve(m.freqs[0], precond="HYBRID", tol=1e-8, maxit=3000)
    names = " ".join(fw.profile())
    fw.set_profiling(False)
    assert r.ok and r.iterations > 0, r
    assert ("cocg_smoother" in names) == smoothed and ("cocg_fwd_sweep_mc" in names) != smoothed, names


def test_other_diagonal_scales_leave_the_coarse_matrices_out(fw):
    """SIGMA_DIAG other than 1 takes the colour sweeps: after an assembly their set-up is six launches (diagonal, lower
    and upper values of the edges; the nodal matrix and its two halves), and no Galerkin matrix among them."""
    m = synth.tidal_box(6, 6, 5, seed=1, half_km=10.0)
    fw.load_model(m)
    fw.set_spmv_rows_per_warp(1)  # no timing runs
    count = []
    for k in range(4):
        if k != 3:  # the third solve after an assembly with buffers and tables at hand, the fourth without one
            fw.assemble()
        before = capi.lib().afem_launch_count()
        fw.solve(m.freqs[0], precond="HYBRID", tol=1e-10, maxit=8, sigma_diag=1.5, use_graph=False)
        count.append(capi.lib().afem_launch_count() - before)
    fw.set_spmv_rows_per_warp(0)
    assert count[2] - count[3] == 6, count
    fw.assemble()  # and back to the smoothed iteration
    assert fw.solve(m.freqs[0], precond="HYBRID", tol=1e-9, maxit=2000).ok


@pytest.mark.parametrize("ns,precision", [(1, "fp64"), (16, "fp64"), (16, "pc32")])
@pytest.mark.parametrize("dims", [(16, 14, 14), (16, 16, 14)])
def test_either_side_of_the_cycles_and_the_launchs_limit(fw, oracle, dims, ns, precision):
    """Level-1 grids of 9 x 8 x 8 = 576 and 9 x 9 x 8 = 648 nodes (one block takes up to 600), and with 16 systems
    430,704 and 490,428 rows x (systems + 2) (one launch takes up to 480,000).  Profiled solves take the launches
    everywhere: the same solution to the tolerance, site fields within 1e-6."""
    m = synth.tidal_box(*dims, seed=8, grf=True, block=False)
    A = oracle.OracleForward(m).assemble(m.freqs[0])
    fw.load_model(m)
    fw.assemble()
    out, its = [], []
    for profiled in (False, True):
        fw.set_profiling(profiled)
        r = fw.solve(np.full(ns, m.freqs[0]), precond="HYBRID", precision=precision, tol=1e-9, maxit=2000)
        fw.set_profiling(False)
        assert r.ok and r.resid_true <= 1e-9, r
        assert oracle.true_residual(A, fw.solution(ns - 1)) <= 1.01e-9
        out.append(fw.sites(m.sites))
        its.append(r.iterations)
    assert abs(its[0] - its[1]) <= 3, its
    assert np.abs(out[0] - out[1]).max() <= 1e-6 * np.abs(out[0]).max()

"""Kernels that serve part of the size range, at the sizes where one hands over to another."""
import numpy as np
import pytest

import oracle
import poissonreconstruction_b200 as prb
from poissonreconstruction_b200 import synthetic
from tests.test_gpu_adaptive import _morton_to_natural_vec, _prolong

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [prb.PR_PRECISION_FP64, prb.PR_PRECISION_MIXED])
@pytest.mark.parametrize("depth,sweeps", [(4, 1), (5, 1), (5, 2), (6, 1)])
def test_coarse_levels_of_the_degree1_vcycle(ctx, depth, sweeps, precision):
    """Depth 4 and two sweeps run the coarse levels one by one, the others in one launch: the solution
    meets the oracle's, and the preconditioner keeps its convergence (a factor of about ten per
    iteration, so at most 15 iterations to 1e-10)."""
    pts = synthetic.torus(3000, seed=40 + depth)
    st = ctx.solve(pts, prb.ReconstructParams(depth=depth, point_weight=4.0, precision=precision,
                                              smooth_sweeps=sweeps, target_rel_residual=1e-10))
    assert st.converged == 1 and st.pcg_iterations <= 15, st
    unit, _ = oracle.to_unit(pts)
    x_ref, _, _ = oracle.Tree(depth, unit).solve_converged(4.0, tol=1e-13, maxit=200000)
    x = ctx.coefficients()
    assert np.linalg.norm(x - x_ref) <= 1e-6 * np.linalg.norm(x_ref)


def _solution(c, pts, params):
    st = c.solve(pts, params)
    return (st.pcg_iterations, st.refinement_steps, st.rel_residual), c.coefficients()


def _same(a, b):
    return a[0] == b[0] and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("precision", [prb.PR_PRECISION_FP64, prb.PR_PRECISION_MIXED])
@pytest.mark.parametrize("depth,pw", [(5, 4.0), (6, 0.0), (7, 4.0)])
def test_coarse_levels_in_one_launch_and_level_by_level(ctx, depth, pw, precision, monkeypatch):
    """The kernel of the levels 16^3, 8^3 and 4^3 does the arithmetic of their own kernels: every bit of a
    solve, and of a packed batch's meshes, is the same with and without it."""
    params = prb.ReconstructParams(depth=depth, point_weight=pw, precision=precision)
    clouds = [synthetic.torus(2000 + 500 * k, seed=30 + k) for k in range(3)]
    runs = []
    for value in ("1", "0"):
        monkeypatch.setenv("PR_COARSE_TAIL", value)
        before = prb.kernel_launches()[0]
        one = _solution(ctx, clouds[0], params)
        runs.append((prb.kernel_launches()[0] - before, one, prb.reconstruct_batch(clouds, [params] * 3)))
    (n1, one1, batch1), (n0, one0, batch0) = runs
    assert n0 > n1 and _same(one1, one0)
    for (m1, s1), (m0, s0) in zip(batch1, batch0):
        assert s1.pcg_iterations == s0.pcg_iterations and s1.iso_value == s0.iso_value
        assert np.array_equal(m1.vertices, m0.vertices) and np.array_equal(m1.triangles, m0.triangles)


def test_replayed_and_plain_launches(monkeypatch):
    """One context takes clouds of several sizes, weights, sweeps, depths, precisions and both degrees until
    it has dropped its 64 graphs, comes back to the first of them again and again, and gives what another
    context gives without graphs."""
    configs = []
    for k in range(60):  # two or three graphs of degree 1, one of degree 2 each
        configs.append((1000 + 700 * (k % 5), prb.ReconstructParams(
            depth=5 + k % 2, degree=1 + (k // 2) % 2, point_weight=0.0 if k % 9 == 5 else 1.0 + 0.5 * k,
            smooth_sweeps=1 + (k % 7 == 4),
            precision=prb.PR_PRECISION_FP64 if k % 3 == 2 else prb.PR_PRECISION_MIXED)))
    order = [i for k in range(len(configs)) for i in (k, 0)] + list(range(len(configs)))
    with prb.Context(0) as replayed, prb.Context(0) as plain:
        expected = {}
        for i in order:
            n, params = configs[i]
            pts = synthetic.torus(n, seed=i)
            if i not in expected:
                monkeypatch.setenv("PR_GRAPHS", "0")
                expected[i] = _solution(plain, pts, params)
                monkeypatch.delenv("PR_GRAPHS")
            assert _same(_solution(replayed, pts, params), expected[i]), (i, configs[i])


@pytest.mark.parametrize("spmv,resid,smooth", [(2, 4, 4), (4, 2, 4), (4, 4, 2), (2, 2, 4), (4, 2, 2), (2, 4, 2)])
def test_plane_counts_of_the_kernel_families_mix(ctx, spmv, resid, smooth, monkeypatch):
    """Two or four planes per thread, by kernel family: the same bits in any mixture."""
    pts, params = synthetic.torus(3000, seed=33), prb.ReconstructParams(depth=6, point_weight=4.0)
    monkeypatch.setenv("PR_ZT", "4")
    expected = _solution(ctx, pts, params)
    for family, value in (("SPMV16", spmv), ("RESID16", resid), ("SMOOTH16", smooth)):
        monkeypatch.setenv("PR_ZT_" + family, str(value))
    assert _same(_solution(ctx, pts, params), expected)


@pytest.mark.parametrize("precision", [prb.PR_PRECISION_FP64, prb.PR_PRECISION_MIXED])
@pytest.mark.parametrize("depth,offset", [(3, 0), (4, 0), (4, 1), (5, 0), (5, 1), (5, 2)])
def test_operator_on_device_vectors(ctx, depth, offset, precision):
    """The tiled operator (depth >= 4, 16-byte aligned vectors) and the per-node one against the oracle;
    offset: the vectors start that many elements past an aligned address."""
    import torch
    pts = synthetic.sphere(2500, seed=50 + depth)
    ctx.solve(pts, prb.ReconstructParams(depth=depth, point_weight=4.0))
    unit, _ = oracle.to_unit(pts)
    t = oracle.Tree(depth, unit)
    t.assemble(4.0)
    dtype = torch.float64 if precision == prb.PR_PRECISION_FP64 else torch.float32
    x = torch.randn(t.n + offset, dtype=dtype, generator=torch.Generator().manual_seed(depth)).cuda()[offset:]
    y = torch.full((t.n + offset,), float("nan"), dtype=dtype, device="cuda")[offset:]
    torch.cuda.synchronize()
    ctx.apply_operator_device(x.data_ptr(), y.data_ptr(), precision)
    ctx.synchronize()
    y_ref = t.spmv(x.double().cpu().numpy())
    err = np.abs(y.double().cpu().numpy() - y_ref).max()
    # 21 products of at most max|A| max|x| each, rounded to 24 or 53 bits
    assert err <= (1e-13 if dtype == torch.float64 else 1e-5) * np.abs(y_ref).max()


@pytest.mark.parametrize("precision", [prb.PR_PRECISION_FP64, prb.PR_PRECISION_MIXED])
def test_operator_takes_the_tiles_from_16_bytes_on(ctx, precision):
    """Vectors that are aligned to 16 bytes and no further take the kernel of the aligned ones: the same
    bits, where the per-node stencil adds in another order."""
    import torch
    depth = 5
    ctx.solve(synthetic.sphere(2500, seed=55), prb.ReconstructParams(depth=depth, point_weight=4.0))
    dtype = torch.float64 if precision == prb.PR_PRECISION_FP64 else torch.float32
    x0 = torch.randn(8 ** depth, dtype=dtype, generator=torch.Generator().manual_seed(5))
    got = {}
    for nbytes in (0, x0.element_size(), 16):
        k = nbytes // x0.element_size()
        x, y = (torch.zeros(8 ** depth + k, dtype=dtype, device="cuda")[k:] for _ in range(2))
        assert x.data_ptr() % 32 == nbytes and y.data_ptr() % 32 == nbytes
        x.copy_(x0)
        torch.cuda.synchronize()
        ctx.apply_operator_device(x.data_ptr(), y.data_ptr(), precision)
        ctx.synchronize()
        got[nbytes] = y.cpu().numpy()
    assert np.array_equal(got[0], got[16])
    assert not np.array_equal(got[0], got[x0.element_size()])


@pytest.mark.parametrize("precision", [prb.PR_PRECISION_FP64, prb.PR_PRECISION_MIXED])
@pytest.mark.parametrize("depth", [5, 6, 7])
def test_degree2_short_plane_runs(ctx, depth, precision):
    """The levels up to 128^3 run in short runs of planes: the solution satisfies the oracle's equations
    to the requested residual (1e-10, times ten for the two operators' own rounding)."""
    pts = synthetic.torus(4000, seed=60 + depth)
    st = ctx.solve(pts, prb.ReconstructParams(depth=depth, degree=2, point_weight=4.0, precision=precision,
                                              target_rel_residual=1e-10))
    assert st.converged == 1 and st.pcg_iterations <= 11, st
    unit, _ = oracle.to_unit(pts)
    t = oracle.Tree2(depth, unit, 4.0)
    b = t.rhs()
    assert np.linalg.norm(b - t.apply(ctx.coefficients())) <= 1e-9 * np.linalg.norm(b)


@pytest.mark.parametrize("depth,n", [(5, 700_001), (6, 50_000), (7, 20_000)])
def test_staged_host_copies(ctx, depth, n):
    """Copies to and from pageable memory on either side of the staging thresholds (32 MiB in; 1 and 8
    MiB out) give the same bytes as copies to and from pinned memory, which are not staged."""
    import torch
    pts = synthetic.sphere(n, seed=70 + depth)
    params = prb.ReconstructParams(depth=depth, point_weight=4.0)
    ctx.solve(pts, params)
    x = ctx.coefficients()
    ctx.solve(torch.from_numpy(pts).pin_memory().numpy(), params)
    y = torch.empty(8 ** depth, dtype=torch.float64).pin_memory().numpy()
    prb._check(prb.lib().pr_ctx_get_coefficients(ctx._h, prb._ptr(y)))
    assert np.array_equal(x, y)


@pytest.mark.parametrize("side,low", [(0, 0.0), (1, 0.0), (2, 0.0), (4, 0.0), (5, 0.0), (8, 0.0), (4, 0.5)])
def test_vertex_table(ctx, side, low):
    """Cubes of raised coefficients in a level field: no slot, a few, slots on both sides of the smallest
    table (1,024 entries for 512 slots, four to a vertex), and the level at the iso value, where vertices
    fall on corners and share keys."""
    depth = 4
    xyz = np.stack(np.meshgrid(*[np.arange(16)] * 3, indexing="ij"), -1).reshape(-1, 3)
    code = sum(((xyz[:, a] >> b) & 1) << (3 * b + a) for a in range(3) for b in range(depth))
    field = np.empty(16 ** 3)
    field[code] = np.where(((xyz >= 4) & (xyz < 4 + side)).all(1), 2.0, low)
    mesh = ctx.extract(field, 0.5, depth=depth)
    v_ref, t_ref = oracle.extract_surface(depth, field, 0.5)
    assert np.array_equal(mesh.vertices, v_ref)
    assert np.array_equal(mesh.triangles, t_ref)


@pytest.mark.parametrize("depth", [4, 5, 6, 7])
@pytest.mark.parametrize("flags", [0, prb.PR_BAND_FULL])
def test_band_coarse_function(ctx, depth, flags):
    """One to four levels above the coarse one (two taps per axis, then two or three), with bricks at the
    faces of the grid or without: the fixed coarse function is the subdivision of the coarse solution (its
    sums of at most 27 terms to 1e-13), and the mesh uses each of its vertices."""
    coarse = 3
    pts = synthetic.torus(4000, seed=80 + depth)
    ctx.solve(pts, prb.ReconstructParams(depth=coarse, degree=2, point_weight=4.0))
    xc = _morton_to_natural_vec(ctx.coefficients(), coarse)
    mesh, st = ctx.reconstruct(pts, prb.ReconstructParams(depth=depth, coarse_depth=coarse, degree=2, point_weight=4.0,
                                                          band_flags=flags))
    assert st.converged == 1 and len(mesh.triangles) > 0
    _, _, codes = ctx.band_info()
    g_all = _prolong(xc, coarse, depth)
    g = ctx.band_vector(2)
    assert np.max(np.abs(g - g_all[prb.band_natural_index(codes, depth)])) <= 1e-13 * np.max(np.abs(g_all))
    t = mesh.triangles.astype(np.int64)
    assert t.max() + 1 == len(mesh.vertices) == len(np.unique(t))


@pytest.mark.parametrize("degree", [1, 2])
@pytest.mark.parametrize("depth", [4, 5])
@pytest.mark.parametrize("lo,hi", [((0, 0, 0), (3, 5, 4)), ((11, 0, 16), (16, 16, 17)), ((0, 15, 0), (99, 99, 99)),
                                   ((13, 14, 15), (99, 99, 99)), ((0, 0, 0), (99, 99, 99))])
def test_block_classification(ctx, degree, depth, lo, hi):
    """Boxes of raised coefficients at the low and the top faces of the grid and across the 16^3 blocks, in
    a level field: the blocks that are told from their extremes
    and those whose corners are formed give the oracle's mesh, with the iso value between the two levels and
    at each of them."""
    res = 1 << depth
    xyz = np.stack(np.meshgrid(*[np.arange(res)] * 3, indexing="ij"), -1).reshape(-1, 3)
    code = sum(((xyz[:, a] >> b) & 1) << (3 * b + a) for a in range(3) for b in range(depth))
    field = np.empty(res ** 3)
    field[code] = np.where(((xyz >= lo) & (xyz < hi)).all(1), 1.0, -0.5)
    ctx.solve(synthetic.sphere(2000, seed=90), prb.ReconstructParams(depth=depth, degree=degree, point_weight=4.0))
    for iso in (0.25, 1.0, -0.5, 0.0, 2.0):
        mesh = ctx.extract(field, iso)
        v_ref, t_ref = (oracle.extract_surface if degree == 1 else oracle.extract_surface2)(depth, field, iso)
        assert np.array_equal(mesh.vertices, v_ref)
        assert np.array_equal(mesh.triangles, t_ref)


@pytest.mark.parametrize("degree,depth,coarse", [(1, 3, 0), (1, 5, 0), (2, 4, 0), (2, 6, 0), (2, 6, 4)])
def test_breakdown_of_conjugate_gradients(ctx, degree, depth, coarse):
    """A screening weight beyond FP32 makes the FP32 operator infinite: the first direction's product with
    it is not a positive number, the iteration stops there with its solution, zero (on a band the coarse
    function).  The same weight in FP64 is solved."""
    pts = synthetic.torus(2000, seed=1)
    params = dict(depth=depth, degree=degree, coarse_depth=coarse, point_weight=1e150)

    def solution():
        return ctx.band_vector(1) if coarse else ctx.coefficients()

    st = ctx.solve(pts, prb.ReconstructParams(precision=prb.PR_PRECISION_MIXED, **params))
    assert (st.converged, st.pcg_iterations) == (0, 0), st
    start = ctx.band_vector(2) if coarse else np.zeros(8 ** depth)
    assert np.isfinite(start).all() and np.array_equal(solution(), start)
    st = ctx.solve(pts, prb.ReconstructParams(precision=prb.PR_PRECISION_FP64, **params))
    assert st.converged == 1 and np.isfinite(solution()).all(), st

"""Kernels at the sizes where their tiling can go wrong (ragged tails, row and
run lengths around a step, one domain, many nodes on one coarse level) against
the CPU oracle or the mathematics (needs a B200)."""
import dataclasses

import numpy as np
import pytest

import oracle
from agipc_learning_b200 import _native as N
from agipc_learning_b200 import synth
from agipc_learning_b200.solver import MasPcg

pytestmark = pytest.mark.gpu

EPS32 = float(np.finfo(np.float32).eps)


def _graph(m, s):
    m.set_graph(s.fem_count, s.node_offset, s.neighbor_start, s.neighbor_num, s.neighbor_list, s.part_map_real,
                s.real_map_part)
    m.set_contacts(s.pairs)


@pytest.mark.parametrize("nt", [1, 31, 32, 33, 129])
def test_element_kernel_tet_counts(nt):
    """Whole and ragged warps of tets, a third of them inverted: triplets
    bit-exact, values to 1e-9 of each tet's largest entry (the bound of the
    full-size test), nothing written past the last tet."""
    import torch
    X, tets = synth.box_mesh(5, 5, 5, 0.01)
    rng = np.random.default_rng(nt)
    x = X + 0.7 * 0.01 * rng.uniform(-1, 1, X.shape)
    tets = tets[rng.permutation(len(tets))[:nt]]
    Di, vol, u, r = oracle.fem_rest_data(tets, X, np.full(nt, 1e5), 0.45)
    g0, R0, C0, V0 = oracle.fem_snk1(tets, x, Di, vol, u, r, 0.01, 3)
    D = lambda a, t: torch.from_numpy(np.ascontiguousarray(a, t)).cuda()  # noqa: E731
    rows = torch.full((10 * nt + 32,), -7, dtype=torch.int32, device="cuda")
    cols = rows.clone()
    vals = torch.full((10 * nt + 32, 9), np.nan, dtype=torch.float64, device="cuda")
    grad = torch.zeros(x.size, dtype=torch.float64, device="cuda")
    a = [D(tets, np.int32), D(x, np.float64), D(Di, np.float64), D(vol, np.float64), D(u, np.float64), D(r, np.float64)]
    p = [t.data_ptr() for t in a]
    torch.cuda.synchronize()
    with MasPcg() as m:
        N.check(m.lib.maspcg_fem_snk1_gradient_hessian(m.h, nt, p[0], len(X), p[1], p[2], p[3], p[4], p[5], 0.01, 3,
                                                       grad.data_ptr(), rows.data_ptr(), cols.data_ptr(),
                                                       vals.data_ptr()), m.h)
    R, C, V = rows.cpu().numpy(), cols.cpu().numpy(), vals.cpu().numpy()
    assert np.array_equal(R[:10 * nt], R0) and np.array_equal(C[:10 * nt], C0)
    assert np.all(R[10 * nt:] == -7) and np.all(C[10 * nt:] == -7) and np.all(np.isnan(V[10 * nt:]))
    d = np.abs(V[:10 * nt] - V0).reshape(nt, 90).max(axis=1)
    assert np.all(d <= 1e-9 * np.abs(V0).reshape(nt, 90).max(axis=1))
    assert np.abs(grad.cpu().numpy().reshape(-1) - g0.reshape(-1)).max() <= 1e-10 * np.abs(g0).max()


def test_element_kernel_degenerate_tets():
    """Rest state, a flattened, a collapsed and a huge tet: finite values that
    match the eigendecomposition to 1e-9 (repeated and zero singular values)."""
    X = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1.0]])
    tets = np.array([[0, 1, 2, 3]], np.int32)
    Di, vol, u, r = oracle.fem_rest_data(tets, X, np.full(1, 1e3), 0.4)
    shapes = [np.eye(3), np.diag([1.0, 1.0, 0.0]), np.diag([1.0, 0.0, 0.0]), np.zeros((3, 3)), 1e3 * np.eye(3),
              np.diag([1.0, 1.0, -1.0]), 1e-9 * np.eye(3)]
    with MasPcg() as m:
        for F in shapes:
            x = X @ F.T
            _, _, _, V0 = oracle.fem_snk1(tets, x, Di, vol, u, r, 0.1)
            _, _, _, V1 = m.fem_snk1(tets, x, Di, vol, u, r, 0.1)
            assert np.all(np.isfinite(V1)), F
            assert np.abs(V1 - V0).max() <= 1e-9 * np.abs(V0).max(), F


def test_element_kernel_skips_bad_tets():
    """A vertex id outside the mesh is refused, the outputs of that tet's own
    slots are left alone and the other tets' are written as without it."""
    import torch
    X, tets = synth.box_mesh(4, 4, 3, 0.01)
    nt = 45
    tets = np.ascontiguousarray(tets[:nt], np.int32)
    bad = [0, 31, 40]
    Di, vol, u, r = oracle.fem_rest_data(tets, X, np.full(nt, 1e5), 0.45)
    _, R0, C0, V0 = oracle.fem_snk1(tets, X, Di, vol, u, r, 0.01)
    tets[bad, [0, 3, 1]] = len(X)
    D = lambda a, t: torch.from_numpy(np.ascontiguousarray(a, t)).cuda()  # noqa: E731
    rows = torch.full((nt, 10), -7, dtype=torch.int32, device="cuda")
    cols, vals = rows.clone(), torch.full((nt, 90), 5.0, dtype=torch.float64, device="cuda")
    grad = torch.zeros(X.size, dtype=torch.float64, device="cuda")
    a = [D(tets, np.int32), D(X, np.float64), D(Di, np.float64), D(vol, np.float64), D(u, np.float64), D(r, np.float64)]
    p = [t.data_ptr() for t in a]
    torch.cuda.synchronize()
    with MasPcg() as m, pytest.raises(RuntimeError, match="vertex id out of range"):
        N.check(m.lib.maspcg_fem_snk1_gradient_hessian(m.h, nt, p[0], len(X), p[1], p[2], p[3], p[4], p[5], 0.01, 0,
                                                       grad.data_ptr(), rows.data_ptr(), cols.data_ptr(),
                                                       vals.data_ptr()), m.h)
    good = np.setdiff1d(np.arange(nt), bad)
    R, C, V = rows.cpu().numpy(), cols.cpu().numpy(), vals.cpu().numpy()
    assert np.all(R[bad] == -7) and np.all(C[bad] == -7) and np.all(V[bad] == 5.0)
    assert np.array_equal(R[good], R0.reshape(nt, 10)[good]) and np.array_equal(C[good], C0.reshape(nt, 10)[good])
    V0 = V0.reshape(nt, 90)
    assert np.all(np.abs(V - V0)[good].max(axis=1) <= 1e-9 * np.abs(V0[good]).max(axis=1))


def test_element_kernel_nearly_singular_projection():
    """Tets whose scaling Hessian has two eigenvalues around 1e-9 of the third and
    of opposite signs, so that its determinant is lost in rounding: the negative
    one is projected out all the same (1e-9 of each tet's largest entry)."""
    rng = np.random.default_rng(0)
    n = 200000
    S = 10.0 ** rng.uniform(-0.6, 0.6, (n, 3))
    u = 10.0 ** rng.uniform(-9.5, -6.5, n)
    S *= ((1 + u * (1 + rng.uniform(-8, 8, n))) / S.prod(axis=1))[:, None] ** (1 / 3)
    S = -np.sort(-S, axis=1)
    J = S.prod(axis=1)
    A = ((2 * J - 1 - u) / J)[:, None, None] * J[:, None, None] ** 2 / (S[:, :, None] * S[:, None, :])
    d = np.arange(3)
    A[:, d, d] = u[:, None] + (J[:, None] / S) ** 2
    w = np.linalg.eigvalsh(A) / np.abs(A).max(axis=(1, 2))[:, None]
    S, u = (a[(w[:, 0] < -2e-9) & (w[:, 1] > 0) & (w[:, 1] < 2e-9)] for a in (S, u))
    n = len(u)
    assert n > 100
    Q = np.linalg.qr(rng.standard_normal((2, n, 3, 3)))[0]
    F = (Q[0] * S[:, None, :]) @ Q[1].transpose(0, 2, 1)
    F *= np.sign(np.linalg.det(F))[:, None, None]
    x = np.concatenate([np.zeros((n, 1, 3)), F.transpose(0, 2, 1)], axis=1).reshape(-1, 3)
    tets = np.arange(4 * n, dtype=np.int32).reshape(n, 4)
    Di, one = np.tile(np.eye(3).reshape(1, 9), (n, 1)), np.ones(n)
    V0 = oracle.fem_snk1(tets, x, Di, one, u, one, 1.0)[3].reshape(n, 90)
    with MasPcg() as m:
        V1 = m.fem_snk1(tets, x, Di, one, u, one, 1.0)[3].reshape(n, 90)
    assert np.all(np.abs(V1 - V0).max(axis=1) <= 1e-9 * np.abs(V0).max(axis=1))


@pytest.mark.parametrize("n,run", [(2, 1), (31, 2), (255, 3), (257, 4), (2303, 5), (2305, 9)])
def test_merge_run_lengths(n, run):
    """Runs around the four-ahead fetch and element counts around a CTA:
    bit-exact (sums in input order)."""
    rng = np.random.default_rng(n)
    k = (n + run - 1) // run
    key = rng.permutation(np.repeat(np.arange(k), run)[:n])
    r, c = (key % 53).astype(np.int32), (53 + key // 53).astype(np.int32)
    v = rng.standard_normal((n, 9))
    ro, co, vo = oracle.convert_triplets(r, c, v)
    with MasPcg() as m:
        rg, cg, vg = m.convert_bcoo(r, c, v)
    assert np.array_equal(rg, ro) and np.array_equal(cg, co) and np.array_equal(vg, vo)


@pytest.mark.parametrize("precision,matrix", [("fp32", "f32"), ("mixed", "f32"), ("mixed", "f32_split"),
                                              ("mixed", "f32_accurate"), ("reference", "f32")])
def test_iteration_product_row_lengths(precision, matrix):
    """Rows of 1 to 40 blocks (around the steps of 8 and 16) and a dense row:
    the iteration's product within the FP32 summation bound (len eps32 per
    row; 1e-12 for the FP64 matrix)."""
    rng = np.random.default_rng(3)
    nb = 97
    rows, cols = [np.arange(nb)], [np.arange(nb)]
    for i in range(nb):
        k = min(i % 40, nb - 1 - i)
        c = i + 1 + rng.permutation(nb - 1 - i)[:k]
        rows.append(np.full(k, i))
        cols.append(c)
    rows, cols = np.concatenate(rows).astype(np.int32), np.concatenate(cols).astype(np.int32)
    vals = rng.standard_normal((len(rows), 9))
    x = rng.standard_normal(3 * nb)
    with MasPcg(preconditioner="none", precision=precision, matrix=matrix) as m:
        m.set_matrix(vals, rows, cols, nb)
        y = m.spmv_working(x)
    f32 = lambda a: np.asarray(a).astype(np.float32).astype(np.float64)  # noqa: E731
    if precision == "reference":
        A, xx, eps = vals, x, 1e-12
    else:
        A, xx, eps = (vals if matrix == "f32_split" else f32(vals)), f32(x), 3 * 100 * EPS32
    ref = oracle.sym_spmv(1.0, A, rows, cols, xx)
    mag = oracle.sym_spmv(1.0, np.abs(A), rows, cols, np.abs(xx))
    assert np.all(np.abs(y - ref) <= eps * mag)


def _islands(n, edge):
    """A box mesh with only every other edge of its neighbour graph kept, so
    that banks fall into many components at every level."""
    s = synth.cube_system(n, E=1e5, seed=7)
    rng = np.random.default_rng(edge)
    keep = rng.random(s.nb) < 0.5
    start, num, lst = s.neighbor_start, s.neighbor_num, s.neighbor_list
    lists = [[u for u in lst[start[v]:start[v] + num[v]] if keep[u] and keep[v]] for v in range(s.nb)]
    s.neighbor_num = np.array([len(q) for q in lists], np.uint32)
    s.neighbor_start = np.concatenate([[0], np.cumsum(s.neighbor_num)[:-1]]).astype(np.uint32)
    s.neighbor_list = np.array([u for q in lists for u in q], np.uint32)
    return s


@pytest.mark.parametrize("precision,inverse", [("reference", "fp32"), ("mixed", "bf16")])
@pytest.mark.parametrize("n", [3, 9, 20])
def test_apply_on_fragmented_hierarchies(n, precision, inverse):
    """Banks of many components (whole levels of short child lists, more nodes
    on a level than a CTA keeps on chip at n = 20) against the oracle's apply
    with the GPU's own inverses: 1e-5, the bound of the FP32 sums."""
    s = _islands(n, n)
    o = oracle.Mas32.from_system(s)
    o.reorder(s.pairs)
    o.prepare_hessian(s.vals, s.rows, s.cols, np.arange(len(s.rows), dtype=np.uint32), 0)
    with MasPcg(precision=precision, inverse=inverse) as m:
        _graph(m, s)
        m.set_matrix(s.vals, s.rows, s.cols, s.nb)
        m.build()
        g64, z = m.domain_matrices(), m.apply_preconditioner(s.b)
        o64, _ = o.domains()
        bound = oracle.Mas32.from_system(s)
        bound.reorder(s.pairs)
        bound.prepare_hessian(np.abs(s.vals), s.rows, s.cols, np.arange(len(s.rows), dtype=np.uint32), 0)
        assert np.all(np.abs(g64 - o64) <= 1e-13 * bound.domains()[0] + 1e-300)
        o.set_inverses(m.domain_inverses())
    zo = o.precondition(s.b)
    assert np.linalg.norm(z - zo) <= 1e-5 * np.linalg.norm(zo)


def _with_outer_rows(s, before, after):
    """The system with rows in front of its FEM range and behind it, each with a
    diagonal block and one that couples it to an FEM row."""
    rng = np.random.default_rng(before + after)
    at = np.concatenate([np.arange(before), before + s.nb + np.arange(after)]).astype(np.int32)
    fem = before + rng.integers(0, s.nb, len(at)).astype(np.int32)
    top = np.abs(s.vals).max()
    vals = np.concatenate([s.vals, np.tile(top * np.eye(3).reshape(1, 9), (len(at), 1)),
                           0.01 * np.abs(s.vals).mean() * rng.standard_normal((len(at), 9))])
    return dataclasses.replace(s, nb=s.nb + len(at), fem_offset=before, vals=vals,
                               rows=np.concatenate([s.rows + before, at, np.minimum(at, fem)]).astype(np.int32),
                               cols=np.concatenate([s.cols + before, at, np.maximum(at, fem)]).astype(np.int32),
                               b=np.concatenate([rng.standard_normal(3 * before), s.b, rng.standard_normal(3 * after)]))


@pytest.mark.parametrize("precision,inverse", [("reference", "fp32"), ("mixed", "bf16"), ("mixed", "fp32")])
@pytest.mark.parametrize("n,before,after", [(9, 0, 0), (9, 5, 7), (20, 1, 33)])
def test_iterates_on_fragmented_hierarchies(n, before, after, precision, inverse):
    """20 iterations of the solve on banks of many components, with rows outside
    the FEM range: the fused restriction, the coarse levels beside or before the
    level-0 apply and r.z from both, against the oracle's iteration with the GPU's
    own inverses.  1e-5: the bound of one FP32 apply's sums, as above."""
    s = _with_outer_rows(_islands(n, n), before, after)
    o = oracle.Mas32.from_system(s)
    o.reorder(s.pairs)
    sel = np.nonzero((s.rows >= before) & (s.cols >= before) & (s.rows < before + s.fem_count) &
                     (s.cols < before + s.fem_count))[0].astype(np.uint32)
    o.prepare_hessian(s.vals, s.rows, s.cols, sel, before)
    with MasPcg(precision=precision, inverse=inverse, gate="euclid", tolerance=1e-30, max_iterations=21) as m:
        _graph(m, s)
        m.set_matrix(s.vals, s.rows, s.cols, s.nb, before)
        m.build()
        o.set_inverses(m.domain_inverses())
        x, res = m.solve(s.b)
    xo, ro = oracle.pcg(s.vals, s.rows, s.cols, s.nb, s.b, precond=oracle.PRECOND_MAS32, gate=oracle.GATE_EUCLID,
                        tol=1e-30, max_iter=21, fem_offset=before, fem_count=s.fem_count, mas=o)
    assert res["iterations"] == ro["iterations"]
    assert np.linalg.norm(x - xo) <= 1e-5 * np.linalg.norm(xo)


@pytest.mark.parametrize("variant", [0, N.FLAG_APPLY_STAGED2, N.FLAG_APPLY_DIRECT])
@pytest.mark.parametrize("inverse", ["bf16", "fp32"])
def test_level_1_beside_level_0(inverse, variant):
    """A fragmented system large enough that the level-0 kernel takes level 1's
    domains (2,662 level-0 domains): 20 iterations against the same with the
    coarse levels on their own, before the level-0 apply.  1e-5: FP32 sums in
    another order."""
    s = _islands(44, 3)
    x = []
    for flags in (variant, variant | N.FLAG_SEQUENTIAL_COARSE):
        with MasPcg(precision="mixed", inverse=inverse, gate="euclid", tolerance=1e-30, max_iterations=21,
                    flags=flags) as m:
            _graph(m, s)
            m.set_matrix(s.vals, s.rows, s.cols, s.nb)
            m.build()
            x.append(m.solve(s.b)[0])
    assert np.linalg.norm(x[0] - x[1]) <= 1e-5 * np.linalg.norm(x[1])


@pytest.mark.parametrize("inverse", ["bf16", "fp16", "fp32"])
def test_coarse_domains_apply_as_level_0(inverse):
    """Without neighbours every vertex is a node of its own on every level, so
    the coarse domains repeat level 0's two, and z is three equal terms; with
    each bank one component and residuals that cancel in it, z is level 0's
    alone.  The two differ by exactly that factor when the coarse levels form a
    domain's product as level 0 does, rounding included."""
    rng = np.random.default_rng(5)
    nb = 64
    rows, cols, vals = [], [], []
    for bank in (0, 32):
        A = rng.standard_normal((96, 96))
        A = A @ A.T / 96 + np.diag(10.0 ** rng.uniform(-2, 2, 96))
        for i in range(32):
            for j in range(i, 32):
                rows.append(bank + i), cols.append(bank + j), vals.append(A[3 * i:3 * i + 3, 3 * j:3 * j + 3].T.reshape(9))
    r = rng.integers(-1000, 1000, (2, 32, 3)).astype(np.float64)
    r[:, 31] -= r.sum(axis=1)
    ident = np.arange(nb, dtype=np.int32)
    chain = [[u for u in (v - 1, v + 1) if 0 <= u < nb and u // 32 == v // 32] for v in range(nb)]
    z = []
    for lists in ([[]] * nb, chain):
        num = np.array([len(q) for q in lists], np.uint32)
        start = (np.cumsum(num) - num).astype(np.uint32)
        with MasPcg(precision="mixed", inverse=inverse) as m:
            m.set_graph(nb, 0, start, num, np.array([u for q in lists for u in q], np.uint32), ident, ident)
            m.set_contacts(np.zeros((0, 4), np.int32))
            m.set_matrix(np.array(vals), np.array(rows, np.int32), np.array(cols, np.int32), nb)
            m.build()
            assert m.info()["levelnum"] == 3
            z.append(m.apply_preconditioner(r.reshape(-1)).astype(np.float32))
    assert np.any(z[1] != 0)
    assert np.array_equal(z[0], z[1] + (z[1] + z[1]))


@pytest.mark.parametrize("n", [1, 33, 2049])
def test_block_gradient_checks_every_index(n):
    """An index outside the system in the last block is refused before anything
    is written; without it the ragged tail is written in full."""
    import torch
    s = synth.cube_system(4, E=1e5, seed=3)
    rng = np.random.default_rng(n)
    r = rng.integers(0, s.nb, n).astype(np.int32)
    c = rng.integers(0, s.nb, n).astype(np.int32)
    lam, x = rng.standard_normal(3 * s.nb), rng.standard_normal(3 * s.nb)
    D = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    with MasPcg(preconditioner="none") as m:
        m.set_matrix(s.vals, s.rows, s.cols, s.nb)
        out = torch.full((n, 9), 5.0, dtype=torch.float64, device="cuda")
        for bad in (s.nb, -1):
            rb = r.copy()
            rb[-1] = bad
            with pytest.raises(RuntimeError):
                m.bcoo_gradient(D(rb), D(c), D(lam), D(x), out)
            assert bool((out == 5.0).all())
        m.bcoo_gradient(D(r), D(c), D(lam), D(x), out)
    L, X = lam.reshape(-1, 3), x.reshape(-1, 3)
    g = -L[r][:, :, None] * X[c][:, None, :]
    g -= np.where((r != c)[:, None, None], X[r][:, :, None] * L[c][:, None, :], 0.0)
    assert np.allclose(out.cpu().numpy(), g.transpose(0, 2, 1).reshape(-1, 9), rtol=1e-14, atol=1e-14)


@pytest.mark.parametrize("precision", ["reference", "mixed"])
@pytest.mark.parametrize("bodies", [1, 3, 4, 5, 16, 17, 33])
def test_body_inverses_and_apply(bodies, precision):
    """12x12 bodies around a CTA's share of them (4 to invert, 16 to apply),
    every other one needing row exchanges: each body's z against a solve, within
    its condition number times eps (FP64; plus z's own rounding in FP32)."""
    rng = np.random.default_rng(bodies)
    nb, rows, cols, vals, dense = 4 * bodies + 5, [], [], [], []
    for k in range(bodies):
        A = rng.standard_normal((12, 12))
        A = A + A.T + (0.0 if k % 2 else 20.0 * np.eye(12))
        if k % 2:
            A[0, 0] = A[3, 3] = 0.0
        dense.append(A)
        for i in range(4):
            for j in range(i, 4):
                rows.append(4 * k + i), cols.append(4 * k + j), vals.append(A[3 * i:3 * i + 3, 3 * j:3 * j + 3].T.reshape(9))
    for i in range(4 * bodies, nb):
        rows.append(i), cols.append(i), vals.append(2.0 * np.eye(3).reshape(9))
    b = rng.standard_normal(3 * nb)
    with MasPcg(preconditioner="block_jacobi", precision=precision) as m:
        m.set_matrix(np.array(vals), np.array(rows, np.int32), np.array(cols, np.int32), nb, 4 * bodies, bodies)
        m.build()
        z = m.apply_preconditioner(b)
    eps = np.finfo(np.float64).eps if precision == "reference" else EPS32
    for k, A in enumerate(dense):
        zk = np.linalg.solve(A, b[12 * k:12 * k + 12])
        tol = 144 * np.finfo(np.float64).eps * np.linalg.cond(A) + 4 * eps * np.linalg.cond(A)
        assert np.linalg.norm(z[12 * k:12 * k + 12] - zk) <= tol * np.linalg.norm(zk), k
    assert np.allclose(z[12 * bodies:], b[12 * bodies:] / 2, rtol=1e-6)


@pytest.mark.parametrize("long_row", [31, 33, 255, 257, 1023, 1024, 1025, 2600])
def test_rows_around_the_bucket_limits(long_row):
    """One row of the given number of triplets (a bucket's sort widths, and the
    limit beyond which a radix sort takes over) among short ones, every third
    triplet repeated: the merge bit-exact, the matrix product to the FP64 bound."""
    rng = np.random.default_rng(long_row)
    nb = 3000
    distinct = nb - 1 - rng.permutation(nb - 8)[:max(long_row * 2 // 3, 1)]
    hub = np.concatenate([distinct, distinct[:long_row - len(distinct)]])
    r = np.concatenate([np.full(long_row, 7), np.arange(nb), rng.integers(0, 7, 500)])
    c = np.concatenate([hub, np.arange(nb), rng.integers(7, nb, 500)])
    order = rng.permutation(len(r))
    r, c = r[order].astype(np.int32), c[order].astype(np.int32)
    v = rng.standard_normal((len(r), 9))
    x = rng.standard_normal(3 * nb)
    ro, co, vo = oracle.convert_triplets(r, c, v)
    with MasPcg(preconditioner="none", precision="reference") as m:
        rg, cg, vg = m.convert_bcoo(r, c, v)
        m.set_matrix(v, r, c, nb)
        y = m.spmv(x)
    assert np.array_equal(rg, ro) and np.array_equal(cg, co) and np.array_equal(vg, vo)
    ref = oracle.sym_spmv(1.0, v, r, c, x)
    mag = oracle.sym_spmv(1.0, np.abs(v), r, c, np.abs(x))
    assert np.all(np.abs(y - ref) <= 3 * 3000 * np.finfo(np.float64).eps * mag + 1e-300)


@pytest.mark.parametrize("last_row", [65597, 65598, 65599, 2 ** 31 - 2])
def test_rows_around_the_bucket_rule(last_row):
    """1,000 triplets in rows up to the last that buckets are kept for (1,000 / 16
    + 65,536 of them), the next two and the largest index: the merge bit-exact,
    and the product of a matrix of as many rows."""
    rng = np.random.default_rng(last_row % 1000)
    n = 1000
    r = np.concatenate([rng.integers(0, 60000, n - 2), [last_row, last_row]]).astype(np.int32)
    c = np.concatenate([rng.integers(60000, 60100, n - 2), [last_row, last_row]]).astype(np.int32)
    r[:300] = r[300:600]  # some repeats
    c[:300] = c[300:600]
    o = rng.permutation(n)
    r, c, v = r[o], c[o], rng.standard_normal((n, 9))
    ro, co, vo = oracle.convert_triplets(r, c, v)
    with MasPcg(preconditioner="none", precision="reference") as m:
        rg, cg, vg = m.convert_bcoo(r, c, v)
        assert np.array_equal(rg, ro) and np.array_equal(cg, co) and np.array_equal(vg, vo)
        if last_row > 70000:
            return
        nb = last_row + 64  # twice the entries: rows around 2,000 / 16 + 65,536
        x = rng.standard_normal(3 * nb)
        m.set_matrix(v, r, c, nb)
        y = m.spmv(x)
    ref, mag = oracle.sym_spmv(1.0, v, r, c, x), oracle.sym_spmv(1.0, np.abs(v), r, c, np.abs(x))
    assert np.all(np.abs(y - ref) <= 3 * n * np.finfo(np.float64).eps * mag)


@pytest.mark.parametrize("where", ["spread", "last"])
def test_long_row_among_many_triplets(where):
    """A row of 5,000 among 700,000 triplets, met in the first or in a later round
    of the counting pass: the merge bit-exact, the product to the FP64 bound."""
    rng = np.random.default_rng(11)
    n, nb = 700000, 60000
    r = rng.integers(0, nb, n)
    at = rng.permutation(n)[:5000] if where == "spread" else np.arange(n - 5000, n)
    r[at] = 77
    c = np.maximum(r, rng.integers(0, nb, n))
    r, c, v = r.astype(np.int32), c.astype(np.int32), rng.standard_normal((n, 9))
    x = rng.standard_normal(3 * nb)
    ro, co, vo = oracle.convert_triplets(r, c, v)
    with MasPcg(preconditioner="none", precision="reference") as m:
        rg, cg, vg = m.convert_bcoo(r, c, v)
        m.set_matrix(v, r, c, nb)
        y = m.spmv(x)
    assert np.array_equal(rg, ro) and np.array_equal(cg, co) and np.array_equal(vg, vo)
    ref, mag = oracle.sym_spmv(1.0, v, r, c, x), oracle.sym_spmv(1.0, np.abs(v), r, c, np.abs(x))
    assert np.all(np.abs(y - ref) <= 3 * 5100 * np.finfo(np.float64).eps * mag)


@pytest.mark.parametrize("inverse", ["fp32", "bf16"])
def test_handles_on_two_devices(inverse):
    """A handle on a second GPU, after one on the first: a kernel's limit of
    shared memory is a device's own.  Solves, and the local checks."""
    import torch
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    s = synth.cube_system(9, E=1e5, seed=1)
    x = []
    for device in (0, 1):
        with torch.cuda.device(device), MasPcg.from_system(s, precision="mixed", inverse=inverse, gate="euclid") as m:
            x.append(m.solve(s.b)[0])
            assert m.local_diagnostics()["matrix_count"] > 0
    assert np.linalg.norm(x[0] - x[1]) <= 1e-6 * np.linalg.norm(x[0])

"""The linear solve's kernel variants at the sizes where each begins and ends.

The system K^T du = g is solved to a relative residual of 1e-11 and checked
against the exported matrix in FP64: the true residual may exceed the
recurrence's by the rounding of the recurrence, eps x iterations x
||A| |x|| / |g| (each iteration's update and product round once at that
scale), so the bound is 1e-11 + 4 eps x iterations x ||A| |x|| / |g|."""
import numpy as np
import pytest

from tissuefolding_paperversion_gb300 import api, mesh

pytestmark = pytest.mark.gpu
RTOL = 1e-11
EPS = np.finfo(np.float64).eps


def _sheet(nx, ny, layers, eta, seed=3):
    rng = np.random.default_rng(seed)
    pos, conn, pl = mesh.rect_sheet(nx + 1, ny + 1, 5.0, layers, 5.0 * layers, 0.5, rng)
    ne, nn = conn.size // 6, pl.size
    fixed = np.zeros((nn, 3), dtype=np.uint8)
    fixed[pl == 0, 2] = 1
    ev = np.zeros((nn, 3))
    ev[pl != 2] = 10.0
    return mesh.Tissue(pos=pos, conn=conn, fixed=fixed.reshape(-1), ext_visc=ev.reshape(-1), node_placement=pl,
                       E=rng.lognormal(np.log(1000.0), 0.3, size=ne), nu=np.full(ne, 0.3), eta=np.full(ne, eta),
                       rates=np.zeros(3 * ne))


def _check_solution(s, out, rows):
    """rows: DOF range of every instance (each is solved to RTOL of its own |g|)."""
    ia, ja, a = s.export_csr(0.0)
    g, du = s.residual(), s.delta_u()
    n = len(ia) - 1
    r = np.repeat(np.arange(n), np.diff(ia))
    Ax = np.bincount(ja, weights=a * du[r], minlength=n)  # A = K^T
    mag = np.bincount(ja, weights=np.abs(a * du[r]), minlength=n)
    for lo, hi in rows:
        ng = np.linalg.norm(g[lo:hi])
        bound = RTOL + 4 * EPS * max(out["iters"], 1) * np.linalg.norm(mag[lo:hi]) / ng
        assert np.linalg.norm((g - Ax)[lo:hi]) <= bound * ng, (lo, hi, out)


def _solve(s, ts):
    states = [mesh.perturbed_state(t, seed=5 + i) for i, t in enumerate(ts)]
    un = np.concatenate([v[1] for v in states])
    s.set_positions(un)
    s.begin_step(ts[0].dt)
    s.set_state(np.concatenate([v[0] for v in states]), un, ts[0].dt)
    s.assemble()
    out = s.solve()
    off = np.cumsum([0] + [3 * t.n_nodes for t in ts])
    _check_solution(s, out, list(zip(off[:-1], off[1:])))
    return out


# levels 48/4 and 243/9 (the coarsest level alone is dense), 507/25/1 (150
# rows: a partly filled group of columns), 6080/286/15, 11163/441/35/1
@pytest.mark.parametrize("eta", [0.0, 100.0])
@pytest.mark.parametrize("nx,ny,layers", [(3, 3, 2), (8, 8, 2), (12, 12, 2), (31, 37, 4), (60, 60, 2)])
def test_multigrid_with_a_dense_coarse_operator(nx, ny, layers, eta):
    t = _sheet(nx, ny, layers, eta)
    with api.Solver(t, precond=2, krylov_rtol=RTOL) as s:
        assert _solve(s, [t])["iters"] < 80


def test_dense_coarse_operators_of_a_ragged_batch():
    ts = [_sheet(3, 3, 2, 0.0), _sheet(12, 13, 2, 0.0, 4), _sheet(8, 8, 1, 0.0, 5), _sheet(25, 9, 3, 0.0, 6)]
    with api.Batch(ts, precond=2, krylov_rtol=RTOL) as s:
        _solve(s, ts)


# The multigrid of the small meshes (auto, atomic assembly) against the general
# path there, block-Jacobi: the same Newton counts, positions to the parity
# tests' 1e-8.  A mesh of 12 nodes has no hierarchy.
@pytest.mark.parametrize("eta", [0.0, 100.0])
@pytest.mark.parametrize("nx,ny,layers,coarsens", [(2, 1, 1, False), (3, 3, 1, True), (9, 7, 3, True), (40, 11, 4, True)])
def test_small_meshes_take_the_multigrid(nx, ny, layers, coarsens, eta):
    t = _sheet(nx, ny, layers, eta)
    t.rates = np.tile([4e-6, 3e-6, 0.0], t.n_elems)
    res = []
    for pc in (0, 1):
        with api.Solver(t, precond=pc) as s:
            s.set_growth_rates(t.rates)
            its = [s.newton_step(t.dt, allow_not_converged=False)["iters"] for _ in range(3)]
            res.append((its, s.positions(), bool(s.multigrid_info()[0])))
    assert res[0][0] == res[1][0]
    assert np.abs(res[0][1] - res[1][1]).max() <= 1e-8 * np.abs(res[1][1]).max()
    assert (res[0][2], res[1][2]) == (coarsens, False)


def test_order_fixed_small_meshes_keep_block_jacobi_for_steps():
    t = _sheet(9, 7, 3, 0.0)
    with api.Solver(t, deterministic=True) as s:
        assert s.multigrid_info()[0] == []
        lv, sv = s.adjoint_forward(np.full(t.n_elems, 1e-6), np.log(t.E), 1, t.dt, 1, np.array([20.0, 20.0, 5.0, 40.0]))
        sv.free()
        assert s.multigrid_info()[0] == []


def test_singular_system_goes_to_block_jacobi():
    """No external viscosity: the in-plane rigid motions have no stiffness.
    Block-Jacobi solves the (consistent) system, the multigrid may not; then
    the handle stays with block-Jacobi."""
    t = _sheet(12, 12, 2, 0.0)
    t.ext_visc[:] = 0.0
    uk, un = mesh.perturbed_state(t, seed=8, amp=0.005)
    res = []
    for pc in (0, 1):
        with api.Solver(t, precond=pc) as s:
            for _ in range(2):
                s.set_state(uk, un, t.dt)
                s.assemble()
                out = s.solve()
                assert out["relres"] <= 1e-8
            res.append(s.residual())
    np.testing.assert_allclose(res[0], res[1], rtol=0, atol=1e-12 * np.abs(res[1]).max())


def test_iteration_cap_is_the_callers():
    t = _sheet(12, 12, 2, 100.0)
    uk, un = mesh.perturbed_state(t, seed=8)
    with api.Solver(t, krylov_max_iter=3) as s:
        s.set_state(uk, un, t.dt)
        s.assemble()
        out = s.solve(allow_not_converged=True)
        assert out["status"] == api.TF_KRYLOV_NOT_CONVERGED and out["iters"] == 3


# The level-0 transfers with the smoothing folded in against the kernels that
# systems with extra blocks use: an added entry of zero between two far nodes
# makes such a system of the same matrix.  Both solve it, with Krylov counts
# within a quarter of each other (the two cycles differ by rounding and the
# tangent's small asymmetry only).  Sizes: one CTA of nodes, its edge, two
# with a remainder, and a coarse level that runs kernel by kernel (forked).
@pytest.mark.parametrize("eta", [0.0, 100.0])
@pytest.mark.parametrize("nx,ny,layers", [(9, 7, 2), (15, 7, 1), (10, 10, 2), (83, 70, 4)])
def test_folded_transfers_match_the_kernels_of_extra_blocks(nx, ny, layers, eta):
    t = _sheet(nx, ny, layers, eta)
    its = []
    for extra in (False, True):
        with api.Solver(t, precond=2, krylov_rtol=RTOL) as s:
            uk, un = mesh.perturbed_state(t, seed=5)
            s.set_positions(un)
            s.begin_step(t.dt)
            s.set_state(uk, un, t.dt)
            s.assemble()
            if extra:
                s.add_K_triplets([0], [3 * (t.n_nodes - 1)], [0.0])
            out = s.solve()
            _check_solution(s, out, [(0, 3 * t.n_nodes)])
            its.append(out["iters"])
    assert abs(its[0] - its[1]) <= 0.25 * its[1] + 1, its


# The element kernel's tile edges: prism counts around multiples of the tiles (8,
# 16, 32), one and several layers, both stiffness paths and both assemblies,
# strongly deformed.  K (FP64 sums of double-float blocks) and g against the
# element routine that the parity tests pin to the oracle (tf_element_eval, FP64),
# summed here: 1e-11 of the largest entry, the parity tests' bound.
@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("eta", [0.0, 100.0])
@pytest.mark.parametrize("nx,ny,layers", [(1, 1, 1), (1, 2, 1), (2, 2, 1), (3, 3, 1), (1, 5, 3), (5, 3, 2), (4, 4, 1)])
def test_element_tiles(nx, ny, layers, eta, deterministic):
    t = _sheet(nx, ny, layers, eta)
    if eta:
        t.eta[::3] = 0.0  # prisms without viscosity among the others
    uk, un = mesh.perturbed_state(t, seed=9, amp=0.8)
    with api.Solver(t, deterministic=deterministic) as s:
        s.set_Fg(mesh.growth_Fg(t, seed=10, amp=0.05))
        s.set_state(uk, un, t.dt)  # no viscosity surfaces yet: element terms only
        s.assemble()
        ia, ja, a = s.export_csr(0.0)
        g = s.residual()
        ev = s.element_eval()
    n = 3 * t.n_nodes
    K, f = np.zeros((n, n)), np.zeros(n)
    free = t.fixed == 0
    for e, nodes in enumerate(t.conn.reshape(-1, 6)):
        dof = (3 * nodes[:, None] + np.arange(3)).reshape(-1)
        K[np.ix_(dof, dof)] += ev["Ke"][e] + ev["Kv"][e]
        f[dof] += (ev["fe"][e] + ev["fv"][e]).reshape(-1)
    K *= free[:, None] & free[None, :]
    K[~free, ~free] = 1.0
    got = np.zeros((n, n))
    got[np.repeat(np.arange(n), np.diff(ia)), ja] = a
    assert np.abs(got - K).max() <= 1e-11 * np.abs(K).max()
    assert np.abs(g - f * free).max() <= 1e-11 * np.abs(f).max()


# Meshes of up to 65,536 nodes share a row among the warps of a 32-node CTA; larger
# ones and order-fixed assemblies have a warp per slice.  Node counts with no,
# one and 31 nodes in the last slice, the largest split mesh and the next, both
# preconditioners, with and without extra blocks.
@pytest.mark.parametrize("eta", [0.0, 100.0])
@pytest.mark.parametrize("precond", [1, 2])
@pytest.mark.parametrize("nodes,nx,ny,layers", [(128, 7, 7, 1), (225, 8, 4, 4), (255, 16, 4, 2)])
def test_split_rows_of_small_meshes(nodes, nx, ny, layers, precond, eta):
    t = _sheet(nx, ny, layers, eta)
    assert t.n_nodes == nodes
    uk, un = mesh.perturbed_state(t, seed=5)
    for deterministic in (False, True):
        for extra in (False, True):
            with api.Solver(t, precond=precond, krylov_rtol=RTOL, deterministic=deterministic) as s:
                s.set_positions(un)
                s.begin_step(t.dt)
                s.set_state(uk, un, t.dt)
                s.assemble()
                if extra:
                    s.add_K_triplets([0, 3 * (nodes - 1)], [3 * (nodes - 1), 0], [1e-3, 1e-3])
                out = s.solve()
                _check_solution(s, out, [(0, 3 * nodes)])


@pytest.mark.parametrize("nodes,nx,ny,layers", [(65536, 127, 127, 3), (65790, 128, 169, 2)])
def test_largest_split_mesh_and_the_next(nodes, nx, ny, layers):
    t = _sheet(nx, ny, layers, 100.0)
    assert t.n_nodes == nodes
    with api.Solver(t, krylov_rtol=RTOL) as s:
        assert _solve(s, [t])["iters"] < 200


def test_split_rows_of_a_ragged_batch():
    ts = [_sheet(3, 3, 2, 100.0), _sheet(12, 13, 2, 100.0, 4), _sheet(7, 7, 1, 100.0, 5), _sheet(16, 4, 2, 100.0, 6)]
    for precond in (1, 2):
        with api.Batch(ts, precond=precond, krylov_rtol=RTOL) as s:
            _solve(s, ts)


# tf_solve_bsr_static, one kernel over all SMs: one row, one group of 32 rows and
# one more, a group more per block (4,865 = 152 x 32 + 1), the largest system, and
# rows of up to 120 blocks (more than shared memory holds).  Ragged unsymmetric
# systems with dominant diagonal blocks; rows 5, 10, .. have a diagonal block only.
@pytest.mark.parametrize("n,most", [(1, 1), (32, 5), (33, 9), (2000, 30), (4865, 27), (9000, 120), (16384, 27)])
def test_static_solve_of_ragged_systems(n, most):
    import ctypes as C

    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    cnt = rng.integers(0, most, size=n)
    cnt[5::5] = 0
    rows = np.repeat(np.arange(n), cnt)
    key = np.unique(np.concatenate([rows * n + rng.integers(0, n, size=rows.size), np.arange(n) * n + np.arange(n)]))
    br, bc = key // n, key % n
    val = rng.uniform(-1.0, 1.0, size=(key.size, 3, 3))
    val[br == bc] += 4.0 * most * np.eye(3)
    rowptr = np.searchsorted(br, np.arange(n + 1)).astype(np.int32)
    b = rng.uniform(-1.0, 1.0, size=3 * n)
    d = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda()
         for k, v in dict(rowptr=rowptr, col=bc.astype(np.int32), val=val.reshape(-1), b=b).items()}
    x = torch.full((3 * n,), float("nan"), dtype=torch.float64, device="cuda")
    it, rr = C.c_int32(0), C.c_double(0.0)
    p = lambda a: C.c_void_p(a.data_ptr())  # noqa: E731
    st = api.load().tf_solve_bsr_static(n, p(d["rowptr"]), p(d["col"]), p(d["val"]), p(d["b"]), p(x), RTOL, 500, None,
                                        C.byref(it), C.byref(rr))
    assert st == api.TF_OK, api.load().tf_last_error().decode()
    assert rr.value <= RTOL
    xs = x.cpu().numpy().reshape(n, 3)
    prod = np.einsum("kij,kj->ki", val, xs[bc])
    Ax, mag = np.zeros((n, 3)), np.zeros((n, 3))
    np.add.at(Ax, br, prod)
    np.add.at(mag, br, np.einsum("kij,kj->ki", np.abs(val), np.abs(xs[bc])))
    nb = np.linalg.norm(b)
    bound = RTOL + 4 * EPS * it.value * np.linalg.norm(mag) / nb
    assert np.linalg.norm(b - Ax.reshape(-1)) <= bound * nb
    # a cap is kept, and the second call does not see the first one's state
    st = api.load().tf_solve_bsr_static(n, p(d["rowptr"]), p(d["col"]), p(d["val"]), p(d["b"]), p(x), 1e-300, 1, None,
                                        C.byref(it), C.byref(rr))
    assert it.value <= 1
    st = api.load().tf_solve_bsr_static(n, p(d["rowptr"]), p(d["col"]), p(d["val"]), p(d["b"]), p(x), RTOL, 500, None,
                                        C.byref(it), C.byref(rr))
    assert st == api.TF_OK and np.array_equal(x.cpu().numpy().reshape(n, 3), xs)  # fixed order of sums


# Coarse images of many extra blocks (a lane group takes five at a time; the warps
# of a split CTA share a row's): a node coupled to 0, 1, 4, 5, 6 and 31 others, its
# CTA's neighbours to none, split and whole rows, both preconditioners.
@pytest.mark.parametrize("precond", [1, 2])
@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("many", [1, 4, 5, 6, 31])
def test_rows_with_many_extra_blocks(many, deterministic, precond):
    t = _sheet(16, 11, 2, 0.0)
    uk, un = mesh.perturbed_state(t, seed=5)
    free = np.flatnonzero(t.fixed.reshape(-1, 3).sum(axis=1) == 0)
    far = free[free > t.n_nodes // 2][:many]
    i, j, v = [], [], []
    for q, n in enumerate(far):  # springs between node free[0] and each of the others
        for d in range(3):
            a, b = 3 * free[0] + d, 3 * n + d
            i += [a, b, a, b]
            j += [a, b, b, a]
            v += [1.0 + q, 1.0 + q, -1.0 - q, -1.0 - q]
    with api.Solver(t, precond=precond, krylov_rtol=RTOL, deterministic=deterministic) as s:
        s.set_positions(un)
        s.begin_step(t.dt)
        s.set_state(uk, un, t.dt)
        s.assemble()
        s.add_K_triplets(i, j, v)
        out = s.solve()
        _check_solution(s, out, [(0, 3 * t.n_nodes)])


# The device loop runs several iterations a round: caps below, at and between its
# rounds are kept exactly, on split and whole rows, in a solve and in a Newton step.
@pytest.mark.parametrize("eta", [0.0, 100.0])
@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("cap", [1, 2, 3, 4, 5, 7])
def test_iteration_caps_between_the_loops_rounds(cap, deterministic, eta):
    t = _sheet(12, 12, 2, eta)
    t.rates = np.tile([4e-6, 3e-6, 0.0], t.n_elems)
    uk, un = mesh.perturbed_state(t, seed=8)
    with api.Solver(t, krylov_max_iter=cap, deterministic=deterministic, precond=1) as s:
        s.set_state(uk, un, t.dt)
        s.assemble()
        out = s.solve(allow_not_converged=True)
        assert out["status"] == api.TF_KRYLOV_NOT_CONVERGED and out["iters"] == cap
    steps = []
    for host in (False, True):  # the host-checked loop: the same, but for the solve the device loop hands back
        with api.Solver(t, krylov_max_iter=cap, deterministic=deterministic, precond=1, host_loops=host) as s:
            s.set_growth_rates(t.rates)
            out = s.newton_step(t.dt)
            steps.append((out["status"], out["iters"], out["krylov_max"]))
    assert steps[0] == steps[1]
    assert steps[0][2] <= cap


# A small sheet grown by a quarter passes near a loss of stability, where the
# multigrid's solves drifted from their recurrence and one run in two took extra
# Newton iterations or ended in a tangled shape (steps 790 to 830).  With the
# residual checked, every step takes at most the 4 Newton iterations it takes with
# block-Jacobi, whatever the rounding of the run.
@pytest.mark.parametrize("run", range(3))
def test_solves_near_a_loss_of_stability_keep_their_residual(run):
    rng = np.random.default_rng(3)
    pos, conn, pl = mesh.rect_sheet(5, 4, 5.0, 8, 40.0, 0.5, rng)
    ne, nn = conn.size // 6, pl.size
    fixed = np.zeros((nn, 3), dtype=np.uint8)
    fixed[pl == 0, 2] = 1
    ev = np.zeros((nn, 3))
    ev[pl != 2] = 10.0
    t = mesh.Tissue(pos=pos, conn=conn, fixed=fixed.reshape(-1), ext_visc=ev.reshape(-1), node_placement=pl,
                    E=1000.0 * rng.uniform(0.98, 1.02, size=ne), nu=np.full(ne, 0.3), eta=np.full(ne, 100.0),
                    rates=np.tile([4.26e-6, 4.26e-6, 0.0], ne))
    with api.Solver(t) as s:
        s.set_growth_rates(t.rates)
        for i in range(900):
            out = s.newton_step(t.dt, allow_not_converged=False)
            assert out["iters"] <= 4, (i, out["dunorm"])


# The static solve where fewer thread blocks than SMs can be resident together: one
# block, a few (their vectors in global memory, several groups of rows a warp),
# and 512, which no GPU of this kind takes together: it then runs with fewer.
@pytest.mark.parametrize("blocks", [1, 3, 17, 60, 512])
@pytest.mark.parametrize("n,most", [(33, 9), (2000, 30), (16384, 27)])
def test_static_solve_on_fewer_blocks(n, most, blocks):
    import ctypes as C

    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    rows = np.repeat(np.arange(n), rng.integers(0, most, size=n))
    key = np.unique(np.concatenate([rows * n + rng.integers(0, n, size=rows.size), np.arange(n) * n + np.arange(n)]))
    br, bc = key // n, key % n
    val = rng.uniform(-1.0, 1.0, size=(key.size, 3, 3))
    val[br == bc] += 4.0 * most * np.eye(3)
    b = rng.uniform(-1.0, 1.0, size=3 * n)
    d = [torch.from_numpy(np.ascontiguousarray(v)).cuda()
         for v in (np.searchsorted(br, np.arange(n + 1)).astype(np.int32), bc.astype(np.int32), val.reshape(-1), b)]
    x = torch.full((3 * n,), float("nan"), dtype=torch.float64, device="cuda")
    it, rr = C.c_int32(0), C.c_double(0.0)
    p = [C.c_void_p(a.data_ptr()) for a in d]
    L = api.load()
    st = L.tf_static_solve_blocks(blocks, 0, n, *p, C.c_void_p(x.data_ptr()), C.c_double(RTOL), 500, None, C.byref(it),
                                  C.byref(rr))
    assert st == api.TF_OK, L.tf_last_error().decode()
    xs = x.cpu().numpy().reshape(n, 3)
    Ax, mag = np.zeros((n, 3)), np.zeros((n, 3))
    np.add.at(Ax, br, np.einsum("kij,kj->ki", val, xs[bc]))
    np.add.at(mag, br, np.einsum("kij,kj->ki", np.abs(val), np.abs(xs[bc])))
    bound = RTOL + 4 * EPS * it.value * np.linalg.norm(mag) / np.linalg.norm(b)
    assert rr.value <= RTOL and np.linalg.norm(b - Ax.reshape(-1)) <= bound * np.linalg.norm(b)


def _bending_sheet():
    """192 viscous prisms in eight layers, the apical half growing half as fast
    again: past some 800 steps it comes near a loss of stability."""
    rng = np.random.default_rng(3)
    pos, conn, pl = mesh.rect_sheet(5, 4, 5.0, 8, 40.0, 0.5, rng)
    ne, nn = conn.size // 6, pl.size
    fixed = np.zeros((nn, 3), dtype=np.uint8)
    fixed[pl == 0, 2] = 1
    ev = np.zeros((nn, 3))
    ev[pl != 2] = 10.0
    t = mesh.Tissue(pos=pos, conn=conn, fixed=fixed.reshape(-1), ext_visc=ev.reshape(-1), node_placement=pl,
                    E=1000.0 * rng.uniform(0.98, 1.02, size=ne), nu=np.full(ne, 0.3), eta=np.full(ne, 100.0),
                    rates=np.zeros(3 * ne))
    g = (0.01 + 0.005 * (t.centroids()[:, 2] >= 20.0)) * 1.02 / mesh.HOUR
    t.rates = np.stack([g, g, np.zeros(ne)], axis=1).reshape(-1)
    return t


# A batch of 20,000 nodes of such sheets keeps the multigrid whatever happens: a
# drifted solve goes on from its own residual, at the 4 Newton iterations a step of
# block-Jacobi (without the check both of two runs ended in non-finite values).
def test_batch_near_a_loss_of_stability_keeps_its_residuals():
    ts = [_bending_sheet() for _ in range(112)]
    with api.Batch(ts) as s:
        assert s.multigrid_info()[0][0] == 20160
        s.set_growth_rates()
        for i in range(840):
            out = s.step(ts[0].dt)
            assert np.all(out["converged"]) and np.max(out["iters"]) <= 4, i


# The multigrid asked for, one sheet: BiCGStab with it diverges at step 811 (as it did
# in every run before, with non-finite values); block-Jacobi then solves the step and
# the handle goes back to the multigrid.
@pytest.mark.parametrize("run", range(2))
def test_multigrid_solves_near_a_loss_of_stability_keep_their_residual(run):
    t = _bending_sheet()
    with api.Solver(t, precond=2) as s:
        s.set_growth_rates(t.rates)
        for i in range(840):
            out = s.newton_step(t.dt, allow_not_converged=False)
            assert out["iters"] <= 4, (i, out["dunorm"])
        assert s.multigrid_info()[0]


@pytest.fixture(scope="module")
def bending_states():
    """Positions and growth of the bending sheet at steps 760, 762, .. 838."""
    t = _bending_sheet()
    out = []
    with api.Solver(t) as s:
        s.set_growth_rates(t.rates)
        for i in range(840):
            s.newton_step(t.dt)
            if i >= 760 and i % 2 == 0:
                out.append((s.positions(), s.get_Fg()[0]))
    return t, out


# Every solve that reports success has the residual it was asked for: at most ten
# times the tolerance, or what the rounding of its iterations leaves at a tight one.
@pytest.mark.parametrize("rtol", [1e-8, 1e-10, 1e-13])
@pytest.mark.parametrize("precond", [0, 2])
def test_residuals_near_a_loss_of_stability_follow_the_tolerance(bending_states, precond, rtol):
    t, states = bending_states
    for x, Fg in states:
        with api.Solver(t, precond=precond, krylov_rtol=rtol) as s:
            s.set_Fg(Fg)
            s.set_positions(x)
            s.set_growth_rates(t.rates)
            s.begin_step(t.dt)
            for _ in range(3):
                s.assemble()
                out = s.solve()
                ia, ja, a = s.export_csr(0.0)
                g, p = s.residual(), a * s.delta_u()[np.repeat(np.arange(3 * t.n_nodes), np.diff(ia))]
                r = np.linalg.norm(g - np.bincount(ja, weights=p, minlength=g.size))
                mag = np.linalg.norm(np.bincount(ja, weights=np.abs(p), minlength=g.size))
                assert r <= max(10 * rtol * np.linalg.norm(g), 4 * EPS * max(out["iters"], 1) * mag)
                s.update()


# A caller's iteration cap that ends the solve with either preconditioner: both are
# tried at the first such solve, later ones cost a single attempt with the one that
# came closer (block-Jacobi on a sheet with displaced nodes, the multigrid on one that grew).
@pytest.mark.parametrize("grown", [False, True])
@pytest.mark.parametrize("eta", [0.0, 100.0])
@pytest.mark.parametrize("cap", [2, 5])
def test_capped_solves_are_not_repeated(cap, eta, grown):
    t = _sheet(20, 20, 2, eta)
    uk, un = mesh.perturbed_state(t, seed=5)
    launches = {}
    for pc in (1, 0):
        with api.Solver(t, krylov_max_iter=cap, precond=pc) as s:
            if grown:
                s.set_growth_rates(np.tile([4e-6, 3e-6, 0.0], t.n_elems))
                s.begin_step(t.dt)
            launches[pc] = []
            for _ in range(3):
                if not grown:
                    s.set_state(uk, un, t.dt)
                s.assemble()
                before = s.launch_count()
                out = s.solve(allow_not_converged=True)
                launches[pc].append(s.launch_count() - before)
                assert out["status"] == api.TF_KRYLOV_NOT_CONVERGED and out["iters"] == cap
            if pc == 0:
                assert bool(s.multigrid_info()[0]) == grown
    assert launches[0][2] <= launches[0][0] - launches[1][2], launches
    if not grown:
        assert launches[0][2] == launches[1][2]


# The element kernel's double-float pairs over FP32's range: moduli from 1e-26 to 1e34
# times those of a tissue, K against the element routine's FP64 sums as in
# test_element_tiles (1e-11 of the largest entry).
@pytest.mark.parametrize("scale", [1e-26, 1e-24, 1e-20, 1e20, 1e34])
@pytest.mark.parametrize("eta", [0.0, 100.0])
def test_element_kernel_over_the_range_of_moduli(eta, scale):
    t = mesh.config_tiny(seed=5, n=4, n_layers=2, eta=eta)
    t.E, t.eta = t.E * scale, t.eta * scale
    uk, un = mesh.perturbed_state(t, seed=9, amp=0.8)
    with api.Solver(t) as s:
        s.set_state(uk, un, t.dt)
        s.assemble()
        ia, ja, a = s.export_csr(0.0)
        ev = s.element_eval()
    n = 3 * t.n_nodes
    K = np.zeros((n, n))
    for e, nodes in enumerate(t.conn.reshape(-1, 6)):
        dof = (3 * nodes[:, None] + np.arange(3)).reshape(-1)
        K[np.ix_(dof, dof)] += ev["Ke"][e] + ev["Kv"][e]
    got = np.zeros((n, n))
    got[np.repeat(np.arange(n), np.diff(ia)), ja] = a
    free = np.flatnonzero(t.fixed == 0)
    d = (got - K)[np.ix_(free, free)]
    assert np.abs(d).max() <= 1e-11 * np.abs(K[np.ix_(free, free)]).max()


@pytest.mark.parametrize("scale", [1e36, 1e40, 1e60, 1e100])
@pytest.mark.parametrize("eta", [0.0, 100.0])
def test_moduli_beyond_the_element_kernels_range_are_reported(eta, scale):
    t = mesh.config_tiny(seed=5, n=4, n_layers=2, eta=eta)
    t.E, t.eta = t.E * scale, t.eta * scale
    uk, un = mesh.perturbed_state(t, seed=9, amp=0.05)
    with api.Solver(t) as s:
        s.set_state(uk, un, t.dt)
        s.assemble()
        with pytest.raises(api.TfError) as e:
            s.solve()
        assert e.value.status == api.TF_NAN_DETECTED


# A small mesh on a device with little memory left gets a handle wherever block-Jacobi
# fits: without a hierarchy, if that does not.
@pytest.mark.parametrize("deterministic", [False, True])
def test_small_meshes_do_without_the_multigrid_where_memory_is_short(deterministic):
    torch = pytest.importorskip("torch")
    t = _sheet(60, 60, 2, 100.0)
    t.rates = np.tile([4e-6, 3e-6, 0.0], t.n_elems)
    lp = np.array([100.0, 100.0, 5.0, 40.0])
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (130 << 20), dtype=torch.uint8, device="cuda")
    try:
        with api.Solver(t, deterministic=deterministic) as s:
            assert s.multigrid_info()[0] == []
            s.set_growth_rates(t.rates)
            s.newton_step(t.dt, allow_not_converged=False)
            if deterministic:  # whose hierarchy is built at the first adjoint call
                _, saved = s.adjoint_forward(np.full(t.n_elems, 1e-6), np.log(t.E), 1, t.dt, 1, lp)
                s.adjoint_backward(saved)
                saved.free()
    finally:
        del hog
        torch.cuda.empty_cache()


def _floating_sheet(nx, ny, layers):
    """No external viscosity: the in-plane rigid motions have no stiffness, and the
    multigrid's coarsest matrix is singular.  The systems are consistent."""
    t = _sheet(nx, ny, layers, 0.0)
    t.ext_visc[:] = 0.0
    t.rates = np.tile([4e-6, 3e-6, 0.0], t.n_elems)
    return t


def _residuals(s, out, rows, rtol=1e-8):
    """Every instance's true residual against the tolerance and its rounding."""
    ia, ja, a = s.export_csr(0.0)
    g, n = s.residual(), len(ia) - 1
    p = a * s.delta_u()[np.repeat(np.arange(n), np.diff(ia))]
    r = g - np.bincount(ja, weights=p, minlength=n)
    mag = np.bincount(ja, weights=np.abs(p), minlength=n)
    for lo, hi in rows:
        assert np.linalg.norm(r[lo:hi]) <= (rtol * np.linalg.norm(g[lo:hi])
                                            + 4 * EPS * max(out["iters"], 1) * np.linalg.norm(mag[lo:hi]))


# A solve that the multigrid does not finish is block-Jacobi's: its du solves the
# assembled system, the handle then shows no hierarchy, and later solves and steps work.
@pytest.mark.parametrize("nx,ny,layers", [(12, 12, 2), (20, 20, 2)])
def test_small_handle_goes_to_block_jacobi_and_stays(nx, ny, layers):
    t = _floating_sheet(nx, ny, layers)
    uk, un = mesh.perturbed_state(t, seed=8, amp=0.005)
    with api.Solver(t) as s:
        assert s.multigrid_info()[0]
        s.set_state(uk, un, t.dt)
        for _ in range(2):
            s.assemble()
            _residuals(s, s.solve(), [(0, 3 * t.n_nodes)])
            assert s.multigrid_info()[0] == []
        s.set_growth_rates(t.rates)
        s.set_positions(t.pos)
        s.newton_step(t.dt, allow_not_converged=False)
        assert s.multigrid_info()[0] == []


def test_batch_goes_to_block_jacobi_with_one_instance():
    ts = [_sheet(9, 7, 2, 0.0), _floating_sheet(12, 12, 2), _sheet(5, 8, 3, 0.0, 4)]
    states = [mesh.perturbed_state(t, seed=8, amp=0.005) for t in ts]
    off = np.cumsum([0] + [3 * t.n_nodes for t in ts])
    with api.Batch(ts) as s:
        assert s.multigrid_info()[0]
        s.set_positions(np.concatenate([v[1] for v in states]))
        s.begin_step(ts[0].dt)
        s.set_state(np.concatenate([v[0] for v in states]), np.concatenate([v[1] for v in states]), ts[0].dt)
        for _ in range(2):
            s.assemble()
            _residuals(s, s.solve(), list(zip(off[:-1], off[1:])))
            assert s.multigrid_info()[0] == []


def test_adjoint_forward_goes_to_block_jacobi():
    """The order-fixed handle takes the multigrid for the adjoint's solves only; the
    loss is that of block-Jacobi to the accuracy of the solves."""
    t = _floating_sheet(12, 12, 2)
    lp, loss = np.array([30.0, 30.0, 5.0, 20.0]), []
    for pc in (0, 1):
        with api.Solver(t, deterministic=True, precond=pc) as s:
            lv, saved = s.adjoint_forward(np.full(t.n_elems, 1e-5), np.log(t.E), 2, t.dt, 1, lp)
            saved.free()
            assert s.multigrid_info()[0] == []
            loss.append(lv)
    assert abs(loss[0] - loss[1]) <= 1e-7 * abs(loss[1])


def test_static_solve_gives_up_on_a_block_that_does_not_come():
    """The thread blocks wait for one more than there are: every wait runs out, the
    call returns an error, and the next call is right."""
    import ctypes as C

    torch = pytest.importorskip("torch")
    n = 100
    d = [torch.from_numpy(v).cuda() for v in (np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32),
                                              np.tile((2.0 * np.eye(3)).reshape(-1), n), np.ones(3 * n))]
    x = torch.zeros(3 * n, dtype=torch.float64, device="cuda")
    it, rr = C.c_int32(7), C.c_double(7.0)
    args = [C.c_void_p(a.data_ptr()) for a in d] + [C.c_void_p(x.data_ptr()), C.c_double(RTOL), 500, None, C.byref(it),
                                                   C.byref(rr)]
    L = api.load()
    assert L.tf_static_solve_blocks(0, 1, n, *args) == api.TF_CUDA_ERROR
    assert "lost each other" in L.tf_last_error().decode() and (it.value, rr.value) == (0, 0.0)
    assert L.tf_static_solve_blocks(0, 0, n, *args) == api.TF_OK
    assert np.array_equal(x.cpu().numpy(), np.full(3 * n, 0.5))


# The form of the FP64 product follows from the rows and the method, so a handle's first
# solve times none: with block-Jacobi it launches what it launches without the autotuner.
@pytest.mark.parametrize("eta", [0.0, 100.0])
@pytest.mark.parametrize("deterministic", [False, True])
def test_first_solve_times_no_forms_of_the_product(deterministic, eta):
    t = _sheet(12, 12, 2, eta)
    uk, un = mesh.perturbed_state(t, seed=5)
    launches = []
    for autotune in (True, False):
        with api.Solver(t, precond=1, krylov_max_iter=4, deterministic=deterministic, autotune=autotune) as s:
            s.set_state(uk, un, t.dt)
            s.assemble()
            before = s.launch_count()
            assert s.solve(allow_not_converged=True)["iters"] == 4
            launches.append(s.launch_count() - before)
            assert s.tiles()["spmv_unroll"] == (4 if deterministic and eta == 0.0 else 2)
    assert launches[0] == launches[1], launches


# A tolerance that no solve reaches, so the caller's cap ends both preconditioners'
# attempts and the multigrid comes closer (it halves the residual: 1e-28 after 80, well
# inside FP32's range).  With a cap of 40 later solves are the multigrid's attempt
# alone; with 80 block-Jacobi still gets its turn.
@pytest.mark.parametrize("cap,both", [(40, False), (80, True)])
def test_block_jacobi_keeps_its_turn_under_large_caps(cap, both):
    t = _sheet(20, 20, 2, 0.0)
    launches = {}
    for pc in (1, 0):
        with api.Solver(t, krylov_rtol=1e-200, krylov_max_iter=cap, precond=pc) as s:
            s.set_growth_rates(np.tile([4e-6, 3e-6, 0.0], t.n_elems))
            s.begin_step(t.dt)
            for _ in range(2):
                s.assemble()
                before = s.launch_count()
                assert s.solve(allow_not_converged=True)["status"] == api.TF_KRYLOV_NOT_CONVERGED
                launches[pc] = s.launch_count() - before
            if pc == 0:
                assert s.multigrid_info()[0]
    # 3 launches an iteration with block-Jacobi, 6 with the multigrid here, 1 every third for
    # the loop: the multigrid's attempt alone is 1.9 times block-Jacobi's, both are 2.9 or more
    assert both == (launches[0] > 2.4 * launches[1]), launches

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

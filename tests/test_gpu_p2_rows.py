"""The quadratic-tet assembly (a warp per element, runs of elements that hand
shared entries on) against the general assembly kernel (colour scatter) and
the residual-only call: meshes below one run, of one run per warp and of
several claims with a partial last run; elements in mesh order and shuffled
(neighbours that share a face, an edge, a corner or nothing); J2 points elastic
and yielding; local numberings rotated element by element.  The two differ in the order of the sums only; the tolerance is
the one of the other parity tests."""
import numpy as np
import pytest

import oracle
import pgfem_gpu as pg
import workloads as wl
from test_gpu_parity import check_K, check_R

pytestmark = pytest.mark.gpu


def _rotate(conn, rng):
    """Every element's nodes by a random even permutation of its corners."""
    edge = {frozenset(v): i for i, v in enumerate([(0, 1), (1, 2), (0, 2), (0, 3), (1, 3), (2, 3)])}
    even = [(0, 1, 2, 3), (1, 2, 0, 3), (2, 0, 1, 3), (1, 0, 3, 2), (2, 3, 0, 1), (3, 2, 1, 0), (0, 2, 3, 1), (0, 3, 1, 2)]
    out = conn.copy()
    for e, k in enumerate(rng.integers(0, len(even), len(conn))):
        c = even[k]
        out[e, :4] = conn[e, list(c)]
        for (i, j), x in {(0, 1): 4, (1, 2): 5, (0, 2): 6, (0, 3): 7, (1, 3): 8, (2, 3): 9}.items():
            out[e, x] = conn[e, 4 + edge[frozenset((c[i], c[j]))]]
    return out


@pytest.mark.parametrize("n,model,mixed", [(1, "j2", False), (2, "he", True), (5, "j2", True), (11, "he", False),
                                           (15, "j2", True)])
def test_matches_general_kernel(gpu, n, model, mixed):
    p = wl.tension(n=n, nne=10, model=model, stretch=0.004, predictor=True)
    rng = np.random.default_rng(n)
    if mixed:
        p.conn = np.ascontiguousarray(_rotate(p.conn[rng.permutation(len(p.conn))], rng))
    p.X = p.X + 0.02 / n * rng.uniform(-1, 1, p.X.shape)
    p.u = p.u + 2e-3 / n * rng.uniform(-1, 1, p.ndof)
    ctx = p.context()
    R, K, st = ctx.assemble_RK(p.u, p.u_presc)
    assert st.ok(), st.as_dict()
    g = p.context()
    g.set_scatter_mode(pg.SCATTER_COLOUR)
    Rg, Kg, st = g.assemble_RK(p.u, p.u_presc)
    assert st.ok()
    check_R(R, Rg)
    check_K(K, Kg, p.Ap)
    R2, K2, _ = ctx.assemble_RK(p.u, p.u_presc)  # a second call on the same context
    check_R(R2, Rg)
    check_K(K2, Kg, p.Ap)
    ctx.close()
    g.close()


@pytest.mark.parametrize("n,three_field", [(2, False), (3, True), (11, False)])
def test_graph_replays_the_call(gpu, n, three_field):
    """The captured call (programmatic launches below 16 MB of K, the second
    stream's fork and join above) equals the direct one; replayed twice."""
    import torch

    p = wl.tension(n=n, nne=10, model="he", stretch=0.004, predictor=True)
    ctx = p.context()
    if three_field:
        ne = len(p.conn)
        ctx.set_three_field(np.full(ne, 3.0), np.full(ne, 1.001))
    R, K, st = ctx.assemble_RK(p.u, p.u_presc)
    assert st.ok()
    d_u = torch.from_numpy(p.u).cuda()
    d_p = torch.from_numpy(p.u_presc).cuda()
    d_R = torch.full((p.ndof,), 7.0, dtype=torch.float64, device="cuda")
    d_K = torch.full((p.nnz,), 7.0, dtype=torch.float64, device="cuda")
    g = ctx.graph_create(d_u.data_ptr(), d_p.data_ptr(), d_R.data_ptr(), d_K.data_ptr())
    s = torch.cuda.current_stream()
    for _ in range(2):
        d_K.fill_(5.0)
        g.launch(s.cuda_stream)
    torch.cuda.synchronize()
    check_R(d_R.cpu().numpy(), R)
    check_K(d_K.cpu().numpy(), K, p.Ap)
    g.destroy()
    ctx.close()


def _perturbed(n, model, seed):
    p = wl.tension(n=n, nne=10, model=model, stretch=0.004, predictor=True)
    rng = np.random.default_rng(seed)
    p.conn = np.ascontiguousarray(_rotate(p.conn[rng.permutation(len(p.conn))], rng))
    p.X = p.X + 0.02 / n * rng.uniform(-1, 1, p.X.shape)
    p.u = p.u + 2e-3 / n * rng.uniform(-1, 1, p.ndof)
    return p, rng


# on 148 SMs of three CTAs: runs of two, four and eight elements (2,058, 6,000 and 13,182 of them)
@pytest.mark.parametrize("model", ["he", "j2"])
@pytest.mark.parametrize("n", [7, 10, 13])
def test_runs_match_general_kernel(gpu, n, model):
    p, _ = _perturbed(n, model, n)
    ctx, g = p.context(), p.context()
    R, K, st = ctx.assemble_RK(p.u, p.u_presc)
    assert st.ok(), st.as_dict()
    g.set_scatter_mode(pg.SCATTER_COLOUR)
    Rg, Kg, st = g.assemble_RK(p.u, p.u_presc)
    assert st.ok()
    check_R(R, Rg)
    check_K(K, Kg, p.Ap)


@pytest.mark.parametrize("model", ["he", "j2"])
@pytest.mark.parametrize("n", [7, 10, 13])
def test_three_field_runs_match_oracle(gpu, n, model):
    p, rng = _perturbed(n, model, n)
    P = 300.0 * rng.uniform(-1, 1, p.ne)
    th = 1.0 + 0.002 * rng.uniform(-1, 1, p.ne)
    ctx = p.context()
    ctx.set_three_field(P, th)
    R, K, st = ctx.assemble_RK(p.u, p.u_presc)
    assert st.ok(), st.as_dict()
    Po, mat = oracle.from_workload(p)
    res = Po.assemble_3f(mat, p.u, P, th, u_presc=p.u_presc, state_n=p.state)
    assert res[0] == 0
    check_R(R, res[1])
    check_K(K, res[2], p.Ap)


@pytest.mark.parametrize("n", [7, 10])
def test_nodes_that_stand_twice_in_an_element(gpu, n):
    """A tenth of the elements have a mid-side node that is one of its corners (their
    Jacobian stays positive at the points)."""
    X, conn, _ = pg.mesh_box_tet(n, 10)
    rng = np.random.default_rng(n)
    for e in np.flatnonzero(rng.random(len(conn)) < 0.1):
        x, c = [(4, 0), (4, 1), (5, 1), (5, 2), (6, 0), (6, 2), (7, 0), (7, 3), (8, 1), (9, 3)][rng.integers(10)]
        conn[e, x] = conn[e, c]
    ids, ndof = pg.generate_dof_ids(conn, len(X), np.zeros(X.shape, dtype=np.int64))
    Ap, Ai = pg.psparse_apai(conn, ids, ndof)
    u = rng.uniform(-1e-4, 1e-4, ndof)
    p = wl.Problem("twice", X, conn, ids, ndof, Ap, Ai, pg.material(pg.MODEL_HE, E=200e3, nu=0.3), u)
    R, K, st = p.context().assemble_RK(u)
    assert st.ok(), st.as_dict()
    Po, mat = oracle.from_workload(p)
    err, Ro, Ko, _ = Po.assemble(mat, u)
    assert err == 0
    check_R(R, Ro)
    check_K(K, Ko, Ap)

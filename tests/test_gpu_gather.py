"""R+K assembly of linear tets by the owners of the rows against the per-node
kernel (colour mode, the general path) over the forms of mesh and supports its
lists distinguish, and the forms that keep the reduction path.

Both evaluate the same closed form in FP64; an entry is a sum of at most some
hundred terms of the size of its row's largest entry, so 1e-12 of that size."""
import numpy as np
import pytest

import oracle
import pgfem_gpu as pg
import workloads as wl

pytestmark = pytest.mark.gpu
TOL = 1e-12


def fan(sub):
    """Tets from the centre of a ball to its surface: an octahedron's faces
    subdivided `sub` times, 8 * 4^sub elements around one node."""
    V = [np.array(v, float) for v in ((1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1))]
    F = [(x, y, z) for x in (0, 1) for y in (2, 3) for z in (4, 5)]
    F = [(a, b, c) if np.linalg.det(np.array([V[a], V[b], V[c]])) > 0 else (b, a, c) for a, b, c in F]
    for _ in range(sub):
        mid, out = {}, []
        for a, b, c in F:
            m = []
            for p, q in ((a, b), (b, c), (c, a)):
                key = (min(p, q), max(p, q))
                if key not in mid:
                    v = V[p] + V[q]
                    mid[key] = len(V)
                    V.append(v / np.linalg.norm(v))
                m.append(mid[key])
            out += [(a, m[0], m[2]), (m[0], b, m[1]), (m[2], m[1], c), (m[0], m[1], m[2])]
        F = out
    X = np.vstack([np.zeros(3), np.array(V)])
    conn = np.array([(0, a + 1, b + 1, c + 1) for a, b, c in F], dtype=np.int32)
    return X, conn


def problem(X, conn, codes, model, Pr=None, seed=0):
    ids, ndof = pg.generate_dof_ids(conn, len(X), codes, Pr)
    Ap, Ai = pg.psparse_apai(conn, ids, ndof)
    rng = np.random.default_rng(seed)
    mat = pg.material(model, E=200e3, nu=0.3, **(dict(sigma_y=250.0, H=2000.0) if model == pg.MODEL_J2 else {}))
    npres = max(0, -int(ids.min()))
    return dict(X=X, conn=conn, ids=ids, ndof=ndof, Ap=Ap, Ai=Ai, mat=mat, npres=npres,
                u=rng.uniform(-2e-3, 2e-3, ndof), pres=rng.uniform(-2e-3, 2e-3, npres))


def context(p):
    return pg.Context(p["X"], p["conn"], p["ids"], p["ndof"], p["Ap"], p["Ai"], p["mat"], npres=p["npres"])


def both(p):
    out = []
    for mode in (pg.SCATTER_ATOMIC, pg.SCATTER_COLOUR):
        ctx = context(p)
        ctx.set_scatter_mode(mode)
        # stale buffers: the owners write every entry
        R, K, st = ctx.assemble_RK(p["u"], p["pres"], R=np.full(p["ndof"], 7.0), K=np.full(ctx.nnz, 7.0))
        assert st.ok()
        s = ctx.get_state(1)
        out.append((R, K, s, ctx.launches_per_assembly()))
    (R, K, s, n), (Rc, Kc, sc, _) = out
    rows = np.repeat(np.arange(p["ndof"]), np.diff(p["Ap"]))
    rmax = np.zeros(p["ndof"])
    np.maximum.at(rmax, rows, np.abs(Kc))
    assert np.all(np.abs(K - Kc) <= TOL * rmax[rows])
    assert np.abs(R - Rc).max() <= TOL * np.abs(Rc).max() * len(p["conn"])
    assert np.abs(s - sc).max() <= TOL
    return n


def box_codes(X, support, seed):
    codes = np.zeros(X.shape, dtype=np.int64)
    if support == "face":
        codes[X[:, 0] == 0.0] = 1
        codes[X[:, 0] == 1.0, 0] = -1
    elif support == "mixed":  # every pattern of fixed, prescribed and free components
        codes = np.random.default_rng(seed).choice([0, 0, 0, 1, -1, -2], size=X.shape).astype(np.int64)
        codes[0], codes[1], codes[2] = [0, 0, 0], [-1, 0, -2], [0, 1, 0]
    return codes


@pytest.mark.parametrize("model", [pg.MODEL_HE, pg.MODEL_J2])
@pytest.mark.parametrize("n,support", [(1, ""), (2, "face"), (3, "mixed"), (5, ""), (5, "mixed")])
def test_boxes(gpu, model, n, support):
    X, conn, _ = pg.mesh_box_tet(n, 4)
    assert both(problem(X, conn, box_codes(X, support, n), model)) == 2


@pytest.mark.parametrize("n", [2, 3, 4])
def test_periodic_boxes(gpu, n):
    """Images share the owner; for two cells an element's nodes share it too."""
    X, conn, Pr = pg.mesh_box_tet(n, 4, periodic=True)
    both(problem(X, conn, np.zeros(X.shape, dtype=np.int64), pg.MODEL_J2, Pr))


def test_one_periodic_cell(gpu):
    """Every node is an image of one: the gradients sum to zero, so R and K are
    zero up to the rounding of terms of the size of the moduli."""
    X, conn, Pr = pg.mesh_box_tet(1, 4, periodic=True)
    p = problem(X, conn, np.zeros(X.shape, dtype=np.int64), pg.MODEL_J2, Pr)
    R, K, st = context(p).assemble_RK(p["u"], R=np.full(p["ndof"], 7.0), K=np.full(9, 7.0))
    assert st.ok() and np.abs(R).max() <= 1e-12 * 200e3 and np.abs(K).max() <= 1e-12 * 200e3 * len(conn)


@pytest.mark.parametrize("sub,launches", [(0, 2), (1, 2), (2, 2), (3, 3)])
def test_valence(gpu, sub, launches):
    """8, 32, 128 incident elements (one round, a full round, four rounds) and
    512, beyond the lists: the reduction path."""
    X, conn = fan(sub)
    assert both(problem(X, conn, np.zeros(X.shape, dtype=np.int64), pg.MODEL_J2)) == launches


def test_other_patterns_keep_the_reduction_path(gpu):
    X, conn, _ = pg.mesh_box_tet(2, 4)
    p = problem(X, conn, np.zeros(X.shape, dtype=np.int64), pg.MODEL_HE)
    # rows wider than the elements couple: every row holds every column
    n = p["ndof"]
    p["Ap"], p["Ai"] = (np.arange(n + 1) * n).astype(np.int32), np.tile(np.arange(n), n).astype(np.int32)
    assert both(p) == 3
    # the x component of the first two nodes tied: DOFs shared by part of a node
    p = problem(X, conn, np.zeros(X.shape, dtype=np.int64), pg.MODEL_HE)
    p["ids"][1] = [3, 4, 5]
    p["ids"][2:] = 6 + np.arange(3 * (len(X) - 2)).reshape(-1, 3)
    p["ids"][0] = [1, 2, 3]
    p["ndof"] = n = int(p["ids"].max())
    p["Ap"], p["Ai"] = (np.arange(n + 1) * n).astype(np.int32), np.tile(np.arange(n), n).astype(np.int32)
    p["u"] = np.random.default_rng(0).uniform(-2e-3, 2e-3, n)
    assert both(p) == 3


@pytest.mark.parametrize("sub", [0, 2, 3])
def test_crystal_plasticity_fan_matches_oracle(gpu, sub):
    X, conn = fan(sub)
    ids, ndof = pg.generate_dof_ids(conn, len(X), np.zeros(X.shape, dtype=np.int64))
    Ap, Ai = pg.psparse_apai(conn, ids, ndof)
    rng = np.random.default_rng(sub)
    q = rng.normal(size=(len(conn), 4))
    R_cp = wl.quat_to_rot(q / np.linalg.norm(q, axis=1)[:, None]).reshape(-1, 9)
    state = np.zeros((len(conn), 10))
    state[:, [0, 4, 8]], state[:, 9] = 1.0, 60.0
    disp = np.zeros(X.shape)
    disp[:, 0] = 1e-3 * X[:, 0]
    u = wl.nodal_to_free(ids, disp + rng.uniform(-1e-4, 1e-4, X.shape))
    p = wl.Problem("fan", X, conn, ids, ndof, Ap, Ai, wl.cp_material(), u, state=state, R_cp=R_cp, dt=0.1)
    R, K, st = p.context().assemble_RK(u, dt=0.1, R=np.full(ndof, 7.0), K=np.full(int(Ap[-1]), 7.0))
    assert st.ok()
    P, mat = oracle.from_workload(p)
    err, Ro, Ko, _ = P.assemble(mat, u, state_n=state, dt=0.1)
    assert err == 0
    # two solves to the 1e-10 local residual: 2 mu 1e-10 against some 100 MPa
    assert np.linalg.norm(R - Ro) <= 1.5e-7 * np.linalg.norm(Ro)
    assert np.linalg.norm(K - Ko) <= 1.5e-7 * np.linalg.norm(Ko)

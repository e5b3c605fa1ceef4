"""Contexts of linear tets on a device that has no room for what speeds them up
(row-owner lists, element records): they are created and assemble by the scatter,
and hold no memory for lists they do not use."""
import numpy as np
import pytest

import pgfem_gpu as pg
import workloads as wl
from test_gpu_gather import box_codes, context, problem

pytestmark = pytest.mark.gpu


def _cp(n, scale):
    X, conn, _ = pg.mesh_box_tet(n, 4)
    ids, ndof = pg.generate_dof_ids(conn, len(X), np.zeros(X.shape, dtype=np.int64))
    Ap, Ai = pg.psparse_apai(conn, ids, ndof)
    q = np.random.default_rng(1).normal(size=(len(conn), 4))
    R = wl.quat_to_rot(q / np.linalg.norm(q, axis=1)[:, None]).reshape(-1, 9) * scale
    return pg.Context(X, conn, ids, ndof, Ap, Ai, wl.cp_material(), R_cp=R)


def test_no_room_for_lists_and_records(gpu):
    import torch
    X, conn, _ = pg.mesh_box_tet(40, 4)
    p = problem(X, conn, box_codes(X, "", 0), pg.MODEL_J2)
    full = context(p)
    R, K, st = full.assemble_RK(p["u"])
    assert st.ok() and full.launches_per_assembly() == 2
    whole = full.device_bytes()
    full.close()
    # what the context needs without lists: its arrays and, meanwhile, the column ids
    need = context_bytes_without_lists(p)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    # 40 MB beside them (allocations come in 2 MB): too little for the 67 MB of element records
    room = need + 4 * len(p["Ai"]) + (40 << 20)
    hold = torch.empty(free - room, dtype=torch.uint8, device="cuda")
    ctx = context(p)
    del hold
    torch.cuda.empty_cache()
    assert ctx.launches_per_assembly() == 3 and ctx.device_bytes() == need < whole
    Rs, Ks, st = ctx.assemble_RK(p["u"])
    assert st.ok()
    assert np.linalg.norm(Rs - R) <= 1e-12 * np.abs(Ks).max() * np.sqrt(len(R))
    assert np.linalg.norm(Ks - K) <= 1e-12 * np.linalg.norm(K)


def context_bytes_without_lists(p):
    """A pattern with one more column per row keeps the scatter; the arrays of the
    context do not depend on the columns."""
    n = 300  # rows that get the extra column: the first nodes'
    q = dict(p)
    Ap, Ai = np.asarray(p["Ap"]), np.asarray(p["Ai"])
    rows, last = [], p["ndof"] - 1
    add = np.zeros(p["ndof"], dtype=np.int64)
    for r in range(n):
        cols = Ai[Ap[r]:Ap[r + 1]]
        assert last not in cols
        rows.append(np.append(cols, last))
        add[r] = 1
    q["Ai"] = np.concatenate(rows + [Ai[Ap[n]:]]).astype(np.int32)
    q["Ap"] = (Ap + np.concatenate([[0], np.cumsum(add)])).astype(np.int32)
    ctx = context(q)
    assert ctx.launches_per_assembly() == 3
    b = ctx.device_bytes()
    ctx.close()
    return b


def test_other_crystal_matrices_keep_no_lists(gpu):
    a, b = _cp(6, 1.0), _cp(6, 1.0 + 1e-6)  # rotations; not orthogonal to 1e-12: the sample-frame kernels
    ne = a.ne
    assert b.device_bytes() <= a.device_bytes() - 52 * 8 * ne - 8 * 4 * ne  # no records, no lists

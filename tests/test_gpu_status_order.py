"""Failure counts that one call leaves and the next read clears: a clear is done
before pgfem_gpu_read_status returns, so that it never takes counts of an assembly
that another stream starts right afterwards."""
import numpy as np
import pytest

import pgfem_gpu as pg
import workloads as wl
from test_gpu_gather import problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("own", [False, True])
def test_clear_precedes_the_next_assembly(gpu, own):
    import torch
    X, conn, _ = pg.mesh_box_tet(2, 4)
    p = problem(X, conn, np.zeros(X.shape, dtype=np.int64), pg.MODEL_HE)
    ctx = pg.Context(p["X"], p["conn"], p["ids"], p["ndof"], p["Ap"], p["Ai"], p["mat"])
    s = torch.cuda.Stream() if own else torch.cuda.default_stream()
    with torch.cuda.stream(s):
        u = torch.from_numpy(wl.nodal_to_free(p["ids"], X * [-1.5, 0.0, 0.0])).cuda()  # F11 = -0.5: all inverted
        R = torch.empty(p["ndof"], dtype=torch.float64, device="cuda")
        K = torch.empty(len(p["Ai"]), dtype=torch.float64, device="cuda")
        for _ in range(200):
            ctx.assemble_RK_device(u.data_ptr(), None, R.data_ptr(), K.data_ptr(), s.cuda_stream or None)
            s.synchronize()
            assert ctx.read_status(clear=True).inverted == len(conn)
    ctx.close()

"""Stream order of the three-field local update: what a caller enqueues on a
stream before pgfem_gpu_three_field_update_device (the increment it reads) and
after it (the assembly that reads P and theta) keeps that order, on the default
stream and on a stream of its own, and so does the device Newton step, which
alternates the two.

The update behind a pause and a copy of u and du on the same stream equals the
host-buffer call at round-off; repeated Newton steps follow the oracle's history
within 1e-9 per entry (solves to 1e-12; an assembly from the previous iterate's
P and theta moves the second entry by 2.5e-6)."""
import numpy as np
import pytest

import oracle
import pgfem_gpu as pg
import workloads as wl
from test_gpu_threefield import _case, _oracle_newton

pytestmark = pytest.mark.gpu


def _stream(own):
    import torch
    return torch.cuda.Stream() if own else torch.cuda.default_stream()


@pytest.mark.parametrize("own", [False, True])
def test_update_follows_the_callers_stream(gpu, own):
    import torch
    p, P, th = _case(seed=2)
    ctx = p.context()
    ctx.set_three_field(P, th)
    du = 1e-3 * np.random.default_rng(4).uniform(-1, 1, p.ndof)
    dP, dth, st = ctx.three_field_increments(p.u, du, p.u_presc)
    assert st.ok()
    hu, hd = (torch.from_numpy(a.copy()).cuda() for a in (p.u, du))
    d_u, d_du = torch.zeros_like(hu), torch.zeros_like(hd)
    d_p = torch.from_numpy(p.u_presc.copy()).cuda()
    out = torch.zeros(2 * p.ne, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    s = _stream(own)
    with torch.cuda.stream(s):
        torch.cuda._sleep(20_000_000)  # some 10 ms, in which an update on another stream would run
        d_u.copy_(hu)
        d_du.copy_(hd)
        for dst in (out.data_ptr(), None):
            r = pg.lib().pgfem_gpu_three_field_update_device(ctx.h, d_u.data_ptr(), d_p.data_ptr(), d_du.data_ptr(),
                                                             dst, s.cuda_stream or None)
            assert r == 0
    if own:
        s.synchronize()
    Pg, thg = ctx.get_three_field()  # waits for an update on the default stream
    torch.cuda.synchronize()
    inc = out.cpu().numpy()
    assert np.abs(inc[:p.ne] - dP).max() <= 1e-13 * np.abs(dP).max()
    assert np.abs(inc[p.ne:] - dth).max() <= 1e-13 * np.abs(dth).max()
    assert np.abs(Pg - (P + dP)).max() <= 1e-13 * np.abs(P + dP).max()
    assert np.abs(thg - (th + dth)).max() <= 1e-13
    ctx.close()


@pytest.mark.parametrize("own", [False, True])
@pytest.mark.parametrize("model", ["he", "j2"])
def test_repeated_newton_steps_match_oracle(gpu, model, own):
    import torch
    if model == "j2":
        p = wl.tension(n=2, nne=10, model="j2", stretch=0.003, predictor=True)
    else:
        p = _case(n=2, seed=3, curve=False)[0]
    P0, th0 = np.zeros(p.ne), np.ones(p.ne)
    Po, mat = oracle.from_workload(p)
    state = p.state if model == "j2" else None
    uo, _, _, ho, ok = _oracle_newton(Po, mat, p.u, p.u_presc, P0, th0, state_n=state)
    assert ok
    ctx = p.context()
    solver = pg.Solver(p.Ap, p.Ai, p.ndof, maxit=20000, kdim=100, tol=1e-12)
    s = _stream(own)
    with torch.cuda.stream(s):
        u0, dp = torch.from_numpy(p.u.copy()).cuda(), torch.from_numpy(p.u_presc.copy()).cuda()
        du = torch.empty_like(u0)
        for _ in range(20):
            ctx.set_three_field(P0, th0)
            ctx.reset_state()
            du.copy_(u0)
            info = solver.newton_step(ctx, du.data_ptr(), dp.data_ptr(), iter_max=15, nor_min=1e-10,
                                      stream=s.cuda_stream or None)
            assert info.converged and not info.lin_failed and info.elem_failures == 0
            h = info.history()
            assert len(h) == len(ho)
            assert np.abs(np.array(h) - np.array(ho)).max() <= 1e-9
        u = du.cpu().numpy()
    assert np.linalg.norm(u - uo) <= 1e-8 * np.linalg.norm(uo)
    ctx.close()

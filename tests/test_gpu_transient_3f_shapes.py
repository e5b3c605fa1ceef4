"""The three-field transient's R+K call at the edges of its point kernel (four
lanes per element, 32 elements per block): element counts that leave a partial
block or a partial warp, every volumetric potential, mid-point rules near both
ends, a context's own element order.  R and K equal the oracle's at the
tolerances of the other three-field tests; the residual-only call, which takes
the general route, counts the same inverted points."""
import numpy as np
import pytest

import oracle
import pgfem_gpu as pg
from test_gpu_parity import check_K, check_R
from test_gpu_threefield import _case

pytestmark = pytest.mark.gpu


def _problem(n, vol_pot, seed):
    p, P, th = _case(n=n, seed=seed, vol_pot=vol_pot)
    us = [f * p.u for f in (1.0, 0.7, 0.4)]
    ps = [f * p.u_presc for f in (1.0, 0.7, 0.4)]
    Ps, ths = [P, 0.6 * P + 5.0, 0.3 * P - 5.0], [th, 1.0 + 0.7 * (th - 1.0), 1.0 + 0.4 * (th - 1.0)]
    ctx = p.context()
    ctx.set_three_field(Ps[0], ths[0])
    ctx.set_three_field_history(Ps[1], ths[1], Ps[2], ths[2])
    return p, us, ps, Ps, ths, ctx


@pytest.mark.parametrize("n,vol_pot,alpha", [(1, 99, 0.5), (2, 2, 0.05), (3, 3, 0.95), (5, 99, 0.3)])
def test_matches_oracle(gpu, n, vol_pot, alpha):
    p, us, ps, Ps, ths, ctx = _problem(n, vol_pot, seed=n)
    dt1, dt0, rho = 0.02, 0.03, 1.0e4
    R, K, st = ctx.assemble_RK_transient(us[0], us[1], us[2], alpha, dt1, dt0, rho, presc=tuple(ps))
    assert st.ok(), st.as_dict()
    Po, mat = oracle.from_workload(p)
    err, Ro, Ko = Po.assemble_3f_transient(mat, us, Ps, ths, alpha, dt1, dt0, rho, presc=tuple(ps))
    assert err == 0
    check_R(R, Ro)
    check_K(K, Ko, p.Ap)
    ctx.close()


@pytest.mark.parametrize("which", [0, 1, 2])
def test_inverted_points_are_counted(gpu, which):
    p, us, ps, Ps, ths, ctx = _problem(3, 99, seed=2)
    us[which] = us[which] + 3.0 * np.random.default_rng(1).uniform(-1, 1, p.ndof)
    a = ctx.assemble_RK_transient(us[0], us[1], us[2], 0.5, 0.02, 0.03, 1.0e4, presc=tuple(ps))[2]
    b = ctx.assemble_RK_transient(us[0], us[1], us[2], 0.5, 0.02, 0.03, 1.0e4, presc=tuple(ps), want_K=False)[2]
    assert a.inverted > 0 and a.as_dict() == b.as_dict()
    ctx.close()

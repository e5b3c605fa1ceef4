"""The network kernels where their tiling changes: fewer rows than a tile, one
row more than a round of slots, more tiles than CTAs, rows at addresses that only
allow single loads and stores (tolerances of test_gpu_mlp.py: the arithmetic is
the same), and gradients repeated bit for bit."""
import numpy as np
import pytest

import mlp_oracle as MO
from test_gpu_mlp import rel, setup_model

pytestmark = pytest.mark.gpu


# one tile, a slot per CTA, a second round of slots on 148 SMs
@pytest.mark.parametrize("n", [1, 31, 127, 129, 128 * 148 + 1, 128 * 444 + 5])
@pytest.mark.parametrize("shift", [0, 1])
def test_predict_device(gpu, n, shift):
    import torch
    m, p, x, t, xm, xs, ys = setup_model(n, seed=n % 7)
    dx = torch.empty(n * 34 + 4, device="cuda")[shift:shift + n * 34]
    dx.copy_(torch.from_numpy(x.ravel()))
    out = torch.full((n * 12 + 8,), 7.0, device="cuda")
    m.predict_device(n, dx.data_ptr(), out[shift:].data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    y = out[shift:shift + n * 12].cpu().numpy().reshape(n, 12)
    assert rel(y, MO.forward(p, x, xm, xs, ys)) <= 1e-3
    rest = torch.cat([out[:shift], out[shift + n * 12:]]).cpu().numpy()
    assert (rest == 7.0).all()


@pytest.mark.parametrize("n", [1, 129, 128 * 148 + 77, 128 * 300])
def test_gradient_copies(gpu, n):
    m, p, x, t, xm, xs, ys = setup_model(n, seed=2)
    loss, g = m.loss_grad(x, t)
    lo, go = MO.loss_grad(p, x, t, xm, xs, ys)
    assert abs(loss - lo) <= 1e-4 * lo
    a, b = MO.unpack(g), MO.unpack(go)
    for name, _ in MO.SHAPES:
        assert rel(a[name], b[name]) <= 2e-3, name
    assert np.array_equal(m.loss_grad(x, t)[1], g)


# one tile more than there are CTAs takes the kernel with three tiles in flight
@pytest.mark.parametrize("n", [1, 128, 129, 128 * 148 - 127, 128 * 148, 128 * 148 + 1])
def test_predict_of_few_rows_equals_that_of_many(gpu, n):
    import torch
    many = 128 * 500
    m, _, x, _, _, _, _ = setup_model(many, seed=3)
    dx = torch.from_numpy(x).cuda()
    y, ym = torch.full((n, 12), 7.0, device="cuda"), torch.empty(many, 12, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    m.predict_device(many, dx.data_ptr(), ym.data_ptr(), st)
    m.predict_device(n, dx.data_ptr(), y.data_ptr(), st)
    assert torch.equal(y, ym[:n])


def test_first_training_call_allocates_no_gradient_copies(gpu):
    import torch
    n = 20000
    nets = [setup_model(n, seed=4) for _ in range(2)]
    x, t = (torch.from_numpy(nets[0][k].astype(np.float32)).cuda() for k in (2, 3))
    used = []
    for net in nets:  # the first call of the process may load code
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        net[0].train_device(n, x.data_ptr(), t.data_ptr(), epochs=1, batch=8192)
        used.append(free - torch.cuda.mem_get_info()[0])
    assert used[1] <= 2 << 20  # the row order and the losses; the copies of 64 tiles take 10 MB

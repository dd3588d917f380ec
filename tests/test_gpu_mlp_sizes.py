"""The scorer's gradient at the edges of its tiles (16 samples a warp, 64 a
block, two blocks per SM) against the torch FP64 restatement, and its buffers
between calls: a gradient call leaves none of itself in the next step."""
import numpy as np
import pytest

from mlp_reference import loss_and_grad
from test_gpu_mlp import GRAD_RTOL, data

pytestmark = pytest.mark.gpu


def _context(seed):
    from remobench_b200.lod import Context
    c = Context(slot_capacity=65536, max_nodes=20_000)
    c.allocate(65536, (0, 0, 0), (1, 1, 1))
    c.mlp_init(seed)
    return c


# one sample to past one and past two rounds of 296 blocks
@pytest.mark.parametrize("n", [1, 7, 15, 16, 17, 63, 64, 65, 1000, 18_944, 18_945, 37_890])
def test_gradient_at_tile_edges(n):
    import torch
    ctx = _context(5)
    x, t = data(n, n)
    xd, td = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    rloss, rg = loss_and_grad(ctx.mlp_params(), x, t)
    for _ in range(2):
        g, loss = ctx.mlp_gradients(xd, td)
        assert abs(loss - rloss) <= 1e-3 * max(1.0, abs(rloss))
        assert np.linalg.norm(g - rg) <= GRAD_RTOL * np.linalg.norm(rg)
    ctx.close()


def test_steps_and_gradients_do_not_mix():
    import torch
    a, b = _context(9), _context(9)
    x, t = data(300, 3)
    xd, td = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    for step in range(5):
        b.mlp_gradients(xd, td)
        la = a.mlp_train_step(xd, td, 3e-3, want_loss=True)
        lb = b.mlp_train_step(xd, td, 3e-3, want_loss=step % 2 == 0)
        assert lb is None or abs(la - lb) <= 1e-4 * max(1.0, abs(la))
        # sums differ by their order alone; Adam's early steps are near lr in size
        assert np.max(np.abs(a.mlp_params() - b.mlp_params())) <= 2e-3 * 3e-3 * (step + 1) + 1e-6
    a.close()
    b.close()


def test_loss_of_an_overflowed_activation():
    """Hidden sums past FP32's range are +infinity, and so is their GELU: the loss
    is infinite, not undefined."""
    import torch
    from mlp_reference import OFF
    ctx = _context(1)
    p = np.zeros(len(ctx.mlp_params()), dtype=np.float32)
    for k in ("W1", "W2"):
        p[OFF[k]:OFF["b" + k[1]]] = 1.0
    p[OFF["W3"]:OFF["W3"] + 64], p[OFF["W3"] + 64:OFF["b3"]] = 1.0, -1.0
    ctx.mlp_set_params(p)
    x = torch.full((3, 16), 3.0e38, device="cuda")
    t = torch.tensor([[0.0, 1.0]], device="cuda").repeat(3, 1)
    assert ctx.mlp_gradients(x, t)[1] == float("inf")
    ctx.close()

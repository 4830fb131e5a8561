"""The V-cycle and its gradient for more vectors than the device runs clusters
of eight blocks at once: the same per vector as in small batches."""
import numpy as np
import pytest
import torch

from arcanefem_gb300 import fem, learned

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def net():
    ctx = fem.Context()
    prob = learned.DiffusionProblem(ctx, n=32, seed=3)
    hier = learned.Hierarchy(32, 5, prob.row_ptr, prob.cols)
    net = learned.MPNN(ctx, hier, layers=4, max_batch=64)
    net.set_params(net.init_params(3, edge_scale=0.02))
    net.set_operator(prob.row_ptr, prob.cols, prob.values)
    yield prob, net
    ctx.close()


@pytest.mark.parametrize("coarse_rows", [0, 300, 2048])
@pytest.mark.parametrize("batch", [31, 36, 37, 64])
def test_large_batches_give_each_vector_its_cycle(net, batch, coarse_rows):
    prob, m = net
    m.set_coarse_rows(coarse_rows)
    gen = torch.Generator(device="cuda").manual_seed(batch)
    r = (torch.randn((batch, prob.mesh.nb_node), generator=gen, device="cuda") * prob.interior).float().contiguous()
    z = m.forward(r)
    for k in range(batch):
        assert torch.equal(z[k], m.forward(r[k].contiguous()).reshape(-1))


def test_large_batches_give_the_mean_gradient(net):
    """The loss is a mean over the pairs: a batch of 64 against its two halves, whose gradients go through BF16
    each on its own (the bounds of the gradient test against the oracle)."""
    prob, m = net
    m.set_coarse_rows(2048)
    gen = torch.Generator(device="cuda").manual_seed(1)
    e = torch.randn((64, prob.mesh.nb_node), generator=gen, device="cuda", dtype=torch.float64) * prob.interior
    r = torch.stack([prob.apply(v.contiguous()) for v in e]).float().contiguous()
    e = e.float().contiguous()
    g, loss = m.gradients(r, e)
    halves = [m.gradients(r[k:k + 32].contiguous(), e[k:k + 32].contiguous()) for k in (0, 32)]
    assert abs(loss - 0.5 * (halves[0][1] + halves[1][1])) <= 1e-6 * abs(loss)
    want = 0.5 * (halves[0][0].double() + halves[1][0].double())
    assert float((g.double() - want).norm()) < 6e-2 * float(want.norm())
    assert np.isfinite(loss)

"""The tensor-core convolutions and weight gradients on grids at the edges of their tiling: one plane
column, columns and runs with remainders, grid rows longer than a 128-position tile, a single z run and
many, a batch that does not fill the CTAs.

Both convolution families round activations to BF16 at the same points and differ in the order of
FP32 sums, which flips a rounding here and there: the bar is the one of the two families' own test."""
import numpy as np
import pytest
import torch

from helpers import rel_l2
from platoanalyze_b200.learned import UNet, init_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nodes,batch", [((4, 4, 4), 1), ((5, 9, 6), 3), ((17, 13, 33), 2), ((9, 5, 150), 1), ((70, 6, 6), 1),
                                         ((33, 34, 35), 2), ((12, 64, 20), 5)])
def test_families_agree(nodes, batch):
    rng = np.random.default_rng(7)
    nn = int(np.prod(nodes))
    inp = torch.tensor(rng.uniform(-1, 1, (batch, nn, 8)), dtype=torch.float32).cuda()
    tgt = torch.tensor(rng.standard_normal((batch, nn, 9)), dtype=torch.float32).cuda()
    got = []
    for kind in (UNet.CONV_TCGEN05, UNet.CONV_MMA_SYNC):
        net = UNet(nodes, batch, conv_kernel=kind)
        net.set_params(init_params(net.num_params, 5))
        out = net.forward(inp).cpu().numpy()
        loss, g = net.loss_and_gradients(inp, tgt, want_grads=True)
        net.check()
        got.append((out, loss, g.cpu().numpy()))
        again, _ = net.loss_and_gradients(inp, tgt)
        assert abs(again - loss) <= 1e-6 * loss and np.array_equal(net.forward(inp).cpu().numpy(), out)
    (a, la, ga), (b, lb, gb) = got
    assert rel_l2(a, b) <= 5e-3 and rel_l2(ga, gb) <= 1e-2 and abs(la - lb) <= 5e-3 * lb


@pytest.mark.parametrize("nodes,batch", [((33, 17, 17), 8), ((20, 33, 33), 3), ((65, 33, 33), 2)])
def test_a_member_does_not_depend_on_its_batch(nodes, batch):
    """A batch large enough for the convolutions that march along z against its members one by one, which are
    not (or, on the largest grid, are in the first layers only): the bar of the families above."""
    rng = np.random.default_rng(9)
    nn = int(np.prod(nodes))
    inp = torch.tensor(rng.uniform(-1, 1, (batch, nn, 8)), dtype=torch.float32).cuda()
    net = UNet(nodes, batch)
    net.set_params(init_params(net.num_params, 5))
    whole = net.forward(inp).cpu().numpy()
    for k in range(batch):
        assert rel_l2(net.forward(inp[k:k + 1].contiguous()).cpu().numpy()[0], whole[k]) <= 5e-3
    net.check()

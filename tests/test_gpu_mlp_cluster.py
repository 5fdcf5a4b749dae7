"""The network chain on clusters of four CTAs against one CTA per tile.

Up to 74 tiles of 128 rows a cluster shares each tile (k_mlp_cluster), beyond
that one CTA has it (k_mlp_chain). Every accumulator sums the same products in
the same order in both, so the same rows must give the same bits, whichever
batch they are in; the loss rows are sums of the same column groups where the
outputs are 64 wide, else within FP32 rounding of 256 terms (256 * 2^-24).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LARGE = 75 * 128


def _pair(nout, depth, batch):
    from lcurve_re_b200.mlp import MLP
    small = MLP(nin=9, nout=nout, depth=depth, batch=batch, seed=3)
    large = MLP(nin=9, nout=nout, depth=depth, batch=LARGE, seed=3)
    return small, large


@pytest.mark.parametrize("nout,depth,rows", [(64, 4, 1), (64, 4, 129), (128, 2, 512),
                                             (192, 3, 300), (256, 5, 640), (64, 1, 128)])
def test_forward_is_the_same(nout, depth, rows):
    import torch
    small, large = _pair(nout, depth, rows)
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.rand(LARGE, 9, generator=g, device="cuda") * 2 - 1
    a = small.forward(x[:rows].contiguous()).clone()
    b = large.forward(x)[:rows]
    torch.cuda.synchronize()
    small.check()
    large.check()
    assert torch.equal(a, b)


@pytest.mark.parametrize("nout,depth,batch", [(64, 4, 128), (64, 4, 74 * 128), (256, 2, 384)])
def test_training_pass_is_the_same(nout, depth, batch):
    import torch
    small, large = _pair(nout, depth, batch)
    g = torch.Generator(device="cuda").manual_seed(batch)
    x = torch.rand(LARGE, 9, generator=g, device="cuda") * 2 - 1
    t = torch.randn(LARGE, nout, generator=g, device="cuda")
    small.forward(x[:batch].contiguous(), train=True, target=t[:batch].contiguous())
    large.forward(x, train=True, target=t)
    torch.cuda.synchronize()
    for l in range(depth):
        assert torch.equal(small.Z[l], large.Z[l][:batch]), l
        assert torch.equal(small.Yt[l], large.Yt[l][:, :batch]), l
    if nout == 64:
        assert torch.equal(small.loss_rows, large.loss_rows[:batch])
    else:
        np.testing.assert_allclose(small.loss_rows.cpu(), large.loss_rows[:batch].cpu(),
                                   rtol=256 * 2.0 ** -24)
    # the backward chain from the same output gradient
    large.G[depth][:batch].copy_(small.G[depth])
    small.backward(sync=False)
    large._target_fused = True
    large.backward(sync=False)
    torch.cuda.synchronize()
    for l in range(depth):
        assert torch.equal(small.G[l], large.G[l][:batch]), l
    small.check()
    large.check()


@pytest.mark.parametrize("nout,depth,batch", [(64, 4, 128), (64, 1, 384), (192, 2, 640),
                                              (256, 5, 4096), (128, 3, 1152)])
def test_gradients_in_two_launches(nout, depth, batch):
    """lcg_mlp_grads against FP64 products of the same BF16 factors: the FP32
    sums of K = batch products are within K 2^-24 of the summed magnitudes
    (tensor-core adds truncate: twice that)."""
    import torch
    from lcurve_re_b200.mlp import MLP
    net = MLP(nin=9, nout=nout, depth=depth, batch=batch, seed=1)
    g = torch.Generator(device="cuda").manual_seed(batch)
    net.x.copy_(torch.rand(net.B, 9, generator=g, device="cuda") * 2 - 1)
    t = torch.randn(net.B, nout, generator=g, device="cuda")
    acc = torch.full((1,), 2.5, dtype=torch.float64, device="cuda")
    for _ in range(2):  # the second pass starts from the first one's gradients
        net.forward(net.x, train=True, target=t)
        net.backward(sync=False, loss_acc=acc)
    net.check()
    tol = 2 * batch * 2.0 ** -24
    for l in range(depth + 1):
        n = net.W[l].shape[0]
        G = net.G[l].double()
        prev = net.x.double() if l == 0 else net.Yt[l - 1].double().T
        ref, mag = G.T @ prev, G.abs().T @ prev.abs()
        assert ((net.dW[l][:n].double() - ref).abs() <= tol * mag + 1e-30).all(), l
        ref, mag = G.sum(0), G.abs().sum(0)
        assert ((net.db[l].double() - ref).abs() <= tol * mag + 1e-30).all(), l
    want = 2.5 + 2 * float(net.loss_rows.double().sum())
    assert abs(float(acc) - want) <= 1e-12 * want

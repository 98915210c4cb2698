"""The layer kernels of the closure network where their row streams change shape: images of one and
two rows (every tile's three rows wrap), runs of rows that end inside and across a CTA's range, several
row segments per image row, batches with fewer rows than CTAs, with more, and with several chunks of rows
per CTA of the weight gradient.  Both tensor-core engines
against the FP64 network with the BF16 roundings of the GPU, to the bounds of
tests/test_gpu_closure.py (forward 1e-4, gradients 1e-3 of the tensor's norm), and the tcgen05 engine's
inference against its training forward.
"""
import numpy as np
import pytest

from oracle.cnn_oracle import CNNOracle
from qgn_fortran_b200.closure import ClosureNet

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


@pytest.mark.parametrize("engine", ["tcgen05-layers", "mma.sync"])
@pytest.mark.parametrize("H,W,layers,batch", [(1, 128, 2, 1), (2, 128, 3, 1), (3, 256, 3, 1), (7, 128, 3, 30),
                                              (5, 384, 2, 11), (50, 128, 3, 3), (160, 128, 2, 1),
                                              (100, 128, 2, 24)])
def test_layers(cuda_ok, H, W, layers, batch, engine):
    import torch
    nz = 3
    net = ClosureNet(nz=nz, H=H, W=W, layers=layers, max_batch=batch, seed=4)
    rng = np.random.default_rng(H + W + batch)
    net.set_weights([(w, rng.standard_normal(b.shape).astype(np.float32) * 0.1 * (np.abs(w).sum(axis=(0, 2)) > 0))
                     for w, b in net.get_weights()])
    net.set_engine(engine)
    x = torch.zeros((batch, H, W, net.cin_p), dtype=torch.bfloat16)
    x[..., :2 * nz] = torch.from_numpy(rng.standard_normal((batch, H, W, 2 * nz))).to(torch.bfloat16)
    y = torch.zeros((batch, H, W, net.cout_p), dtype=torch.float32)
    y[..., :nz] = torch.from_numpy(rng.standard_normal((batch, H, W, nz)))
    xd, yd, out = x.cuda(), y.cuda(), torch.zeros_like(y).cuda()
    net.forward(xd, out, batch)
    net.check()
    m = CNNOracle(net.get_weights(), nz)
    want = m.forward(x.float().numpy())[0]
    assert rel(out.cpu().numpy(), want) <= 1e-4
    loss, grads = net.gradients(xd, yd, batch)
    wloss, wgrads = m.loss_and_grads(x.float().numpy(), y.numpy())
    assert loss == pytest.approx(wloss, rel=1e-4)
    for (gw, gb), (ww, wb) in zip(grads, wgrads):
        assert rel(gw, ww) <= 1e-3
        assert rel(gb, wb) <= 1e-3


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
def test_target_of_any_alignment(cuda_ok, offset):
    """The loss kernel reads 16 bytes of the target at a time; a target at any float gives the same bytes."""
    import torch
    nz, H, W, batch = 2, 4, 128, 2
    net = ClosureNet(nz=nz, H=H, W=W, layers=2, max_batch=batch, seed=1)
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn((batch, H, W, net.cin_p), generator=g, device="cuda").to(torch.bfloat16)
    y = torch.randn((batch, H, W, net.cout_p), generator=g, device="cuda")
    buf = torch.zeros(y.numel() + 4, device="cuda")
    moved = buf[offset:offset + y.numel()].view(y.shape)
    moved.copy_(y)
    assert moved.data_ptr() % 16 == 4 * offset
    loss, grads = net.gradients(x, moved, batch)
    want, wgrads = net.gradients(x, y, batch)
    assert loss == want
    for (gw, gb), (ww, wb) in zip(grads, wgrads):
        assert np.array_equal(gw, ww) and np.array_equal(gb, wb)

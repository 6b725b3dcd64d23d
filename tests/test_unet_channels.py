"""Channel counts beyond the tensor-core kernels' shared memory: refused,
forward and backward alike, and taken with set_tcgen05 off."""
import numpy as np
import pytest

from ekcases import rel_l2
from ekman_bl_gb300.duct import EkError
from oracle.unet_ref import Net, layer_specs

EK_ERR_CUDA = 2


def exact_case(C, n, h, w):
    """Weights of a few +-1 an output and small whole inputs: every sum of the
    forward and input-gradient passes is exact in FP32, whatever its order, so
    the same values are rounded to BF16 everywhere."""
    rng = np.random.default_rng(C)
    parts = []
    for ci, co, *_ in layer_specs(2, C):
        wt = np.zeros((co, 9 * ci), np.float32)
        for r in wt:
            r[rng.choice(9 * ci, 3, replace=False)] = rng.choice([-1, 1, 1], 3)
        parts += [wt.ravel(), rng.integers(0, 2, co).astype(np.float32)]
    x = rng.integers(-4, 5, (n, h, w, 2)).astype(np.float32)
    return np.concatenate(parts), x, rng.integers(-4, 5, (n, h, w)).astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("C,h,w,hv,wv", [(48, 8, 8, 8, 8), (48, 8, 264, 8, 256), (64, 16, 40, 16, 32)])
def test_wide_networks(C, h, w, hv, wv):
    import torch
    from ekman_bl_gb300.duct import UNet
    p, x, t = exact_case(C, 1, h, w)
    xd, td = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    net = UNet(2, C, 1, h, w)
    net.set_params(p)
    y = torch.zeros((1, h, w), device="cuda")
    for call in (lambda: net.forward(xd.data_ptr(), 1, y.data_ptr()),
                 lambda: net.gradient(xd.data_ptr(), td.data_ptr(), 1, hv, wv),
                 lambda: net.train_step(xd.data_ptr(), td.data_ptr(), 1, hv, wv, 1e-3)):
        with pytest.raises(EkError) as e:
            call()
        assert e.value.code == EK_ERR_CUDA and "shared memory" in str(e.value)
    assert np.array_equal(net.get_params(), p)
    net.set_tcgen05(False)
    loss, g = net.gradient(xd.data_ptr(), td.data_ptr(), 1, hv, wv, y.data_ptr())
    rloss, ry, rg = Net(p, 2, C, bf16_round=True).loss_and_grads(x, t, hv, wv)
    assert np.array_equal(y.cpu().numpy(), ry.astype(np.float32)) and np.abs(ry).max() > 0
    # sums of P products in another FP32 order: each within about
    # sqrt(P/2) 2^-24 of its size
    tol = 4 * np.sqrt(h * w) * 2.0 ** -24
    assert abs(loss - rloss) <= tol * rloss and rel_l2(g, rg) <= tol

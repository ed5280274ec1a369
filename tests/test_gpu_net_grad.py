"""Loss, mask sum and gradients of the update network around the edges of their reductions."""
import numpy as np
import pytest

import tomo

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    return built_lib


def inputs(B, H, W, seed=3):
    import torch

    g = torch.Generator().manual_seed(seed)
    feat = torch.rand(B, 3, H, W, generator=g) - 0.5
    tgt = 0.02 * torch.randn(B, H, W, generator=g)
    msk = torch.rand(B, H, W, generator=g) * (torch.rand(B, H, W, generator=g) < 0.3)
    return feat.cuda(), tgt.cuda(), msk.cuda()


@pytest.mark.parametrize("shape", [(1, 1, 64), (1, 33, 64), (3, 70, 128), (2, 301, 320), (5, 256, 192)])
def test_loss_and_mask_sum(shape):
    """FP64 sums of the same FP32 terms: order changes the last bits only (1e-12)."""
    import torch

    B, H, W = shape
    feat, tgt, msk = inputs(B, H, W)
    out = torch.empty(B, H, W, device="cuda")
    torch.cuda.synchronize()
    net = tomo.Net()
    net.forward_device(feat.data_ptr(), B, H, W, out.data_ptr())
    grad, loss = net.grad_device(feat.data_ptr(), tgt.data_ptr(), msk.data_ptr(), B, H, W)
    e = ((out - tgt) * msk).cpu().numpy().astype(np.float64)
    want = float((e * e).sum() / msk.cpu().numpy().astype(np.float64).sum())
    assert abs(loss - want) <= 1e-12 * want
    assert np.isfinite(grad).all()


def test_empty_mask_is_refused_and_changes_nothing():
    import torch

    B, H, W = 2, 40, 64
    feat, tgt, msk = inputs(B, H, W)
    none = torch.zeros_like(msk)
    torch.cuda.synchronize()
    net = tomo.Net()
    before = net.params()
    want = net.grad_device(feat.data_ptr(), tgt.data_ptr(), msk.data_ptr(), B, H, W)
    for call in (net.grad_device, net.train_step_device):
        for m in (none, -msk, torch.full_like(msk, float("nan"))):
            torch.cuda.synchronize()
            with pytest.raises(tomo.TomoError) as e:
                call(feat.data_ptr(), tgt.data_ptr(), m.data_ptr(), B, H, W, *((1e-3,) if call == net.train_step_device else ()))
            assert e.value.status == tomo.ERR_ARG
    assert np.array_equal(net.params(), before)
    got = net.grad_device(feat.data_ptr(), tgt.data_ptr(), msk.data_ptr(), B, H, W)
    assert np.array_equal(got[0], want[0]) and got[1] == want[1]


@pytest.mark.parametrize("shape", [(1, 1, 64), (1, 2, 64), (3, 3, 192), (2, 17, 128), (1, 41, 320)])
def test_layers_match_reference(shape):
    """Strips of one row, of fewer rows than the accumulator ring and of more, one column tile and several with a
    part of the last; the bars of the network's other comparisons with the reference (BF16 roundings that flip)."""
    import torch

    import cnn_oracle as K

    def rel(a, b):
        return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-300))

    B, H, W = shape
    feat, tgt, msk = inputs(B, H, W, seed=11)
    out = torch.empty(B, H, W, device="cuda")
    torch.cuda.synchronize()
    net = tomo.Net(0, seed=3)
    p = net.params()
    p[-1] = 0.01
    net.set_params(p)
    net.forward_device(feat.data_ptr(), B, H, W, out.data_ptr())
    grad, loss = net.grad_device(feat.data_ptr(), tgt.data_ptr(), msk.data_ptr(), B, H, W)
    f64, f, t, m = p.astype(np.float64), feat.cpu().numpy().astype(np.float64), tgt.cpu().numpy(), msk.cpu().numpy()
    assert rel(out.cpu().numpy(), K.forward(f64, f, emulate=True)[0]) <= 5e-3
    loss_ref, g_ref = K.loss_and_grad(f64, f, t, m, emulate=True)
    assert abs(loss - loss_ref) <= 1e-2 * loss_ref
    o = 0
    for name, shp in K.SHAPES:
        n = int(np.prod(shp))
        if np.linalg.norm(g_ref[o:o + n]) > 0:
            assert rel(grad[o:o + n], g_ref[o:o + n]) <= 2e-2, name
        o += n

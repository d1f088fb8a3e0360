"""CUDA kernels of the coarse-correction CNN against the numpy restatement
(oracle/cnn_oracle.py): forward output and all four weight gradients, and a
training run that lowers the loss."""
import numpy as np
import pytest

from samrai_b200 import fac
from oracle import cnn_oracle as co

pytestmark = pytest.mark.gpu

S = fac.CNN_BOX


def rel(a, b):
    return float(np.linalg.norm((a - b).ravel()) / max(np.linalg.norm(b.ravel()), 1e-30))


def test_forward_and_gradients_match_oracle(require_gpu):
    import torch
    rng = np.random.default_rng(0)
    n = 2
    ref = co.CNN.init(seed=3)
    x = rng.standard_normal((n, S, S, S)).astype(np.float32)
    t = rng.standard_normal((n, S, S, S)).astype(np.float32)
    mask = np.zeros_like(t)
    mask[:, 1:-1, 1:-1, 1:-1] = 1.0
    net = fac.CNN(max_batch=4)
    net.set_weights(ref.w)
    xd, td, md = (torch.from_numpy(a).cuda() for a in (x, t, mask))
    yd = torch.zeros_like(xd)
    net.forward(xd.data_ptr(), n, yd.data_ptr())
    y_ref, _ = ref.forward(x)
    assert rel(yd.cpu().numpy(), y_ref) < 1e-2
    loss, gs = net.gradients(xd.data_ptr(), td.data_ptr(), md.data_ptr(), n)
    loss_ref, gs_ref = ref.loss_and_grads(x, t, mask)
    assert abs(loss - loss_ref) <= 1e-2 * loss_ref
    for g, gr in zip(gs, gs_ref):
        assert rel(g, gr) < 3e-2, rel(g, gr)
    net.close()


def test_training_lowers_loss(require_gpu):
    import torch
    rng = np.random.default_rng(1)
    n = 8
    # target: a fixed local linear map of the input (a 7-point average)
    x = rng.standard_normal((n, S, S, S)).astype(np.float32)
    t = x.copy()
    for ax in (1, 2, 3):
        t += np.roll(x, 1, axis=ax) + np.roll(x, -1, axis=ax)
    t /= 7.0
    mask = np.zeros_like(t)
    mask[:, 2:-2, 2:-2, 2:-2] = 1.0
    net = fac.CNN(max_batch=n, seed=5)
    xd, td, md = (torch.from_numpy(a).cuda() for a in (x, t, mask))
    losses = [net.train_step(xd.data_ptr(), td.data_ptr(), md.data_ptr(), n, mask.sum(), 3e-3)
              for _ in range(150)]
    assert losses[-1] < 0.3 * losses[0], (losses[0], losses[-1])
    net.close()


def test_batch_walk_matches_single_samples(require_gpu):
    """A batch of many samples (each CTA of the tensor-core convolution walks
    several slabs, its accumulator barrier changing phase between them) gives
    bit for bit what the same samples give alone."""
    import torch
    rng = np.random.default_rng(2)
    n = 160
    net = fac.CNN(max_batch=n, seed=7)
    x = torch.from_numpy(rng.standard_normal((n, S, S, S)).astype(np.float32)).cuda()
    y = torch.zeros_like(x)
    net.forward(x.data_ptr(), n, y.data_ptr())
    for first in (0, 77, n - 2):
        xs = x[first:first + 2].contiguous()
        ys = torch.zeros_like(xs)
        net.forward(xs.data_ptr(), 2, ys.data_ptr())
        assert torch.equal(ys, y[first:first + 2])
    assert torch.isfinite(y).all()
    net.close()


@pytest.mark.parametrize("n", [1, 3])
def test_fractional_masks_match_oracle(n, require_gpu):
    """Masks that are no 0/1 fields (their sum is formed on the device), on
    data of two scales; the bounds of the test above."""
    import torch
    rng = np.random.default_rng(10 + n)
    ref = co.CNN.init(seed=4)
    x = rng.standard_normal((n, S, S, S)).astype(np.float32)
    t = (1e-3 * rng.standard_normal((n, S, S, S))).astype(np.float32)
    mask = rng.random((n, S, S, S)).astype(np.float32)
    net = fac.CNN(max_batch=n)
    net.set_weights(ref.w)
    xd, td, md = (torch.from_numpy(a).cuda() for a in (x, t, mask))
    loss, gs = net.gradients(xd.data_ptr(), td.data_ptr(), md.data_ptr(), n)
    loss_ref, gs_ref = ref.loss_and_grads(x, t, mask)
    assert abs(loss - loss_ref) <= 1e-2 * loss_ref
    for g, gr in zip(gs, gs_ref):
        assert rel(g, gr) < 3e-2, rel(g, gr)
    with pytest.raises(fac.FacError):
        net.gradients(xd.data_ptr(), td.data_ptr(), torch.zeros_like(md).data_ptr(), n)
    net.close()


@pytest.mark.parametrize("n", [25, 130])
def test_walks_of_several_slabs_match_fp64(n, require_gpu):
    """Batches whose slabs (six a sample) exceed the CTAs of the kernels, so
    that a CTA walks several: output, loss and gradients against the network
    in FP64, with the bounds of the oracle test (BF16 weights and activations,
    2^-9 each, through four layers)."""
    import torch
    conv = torch.nn.functional.conv3d
    g = torch.Generator(device="cpu").manual_seed(n)
    x, t = (torch.randn((n, S, S, S), generator=g).cuda() for _ in range(2))
    m = (torch.rand((n, S, S, S), generator=g) < 0.5).float().cuda()
    net = fac.CNN(max_batch=n, seed=9)
    ws = [torch.from_numpy(w).cuda().double().reshape(s).requires_grad_() for w, s in
          zip(net.get_weights(), [(27, 1, 16), (27, 16, 16), (27, 16, 16), (27, 16, 1)])]
    y_ref, loss_ref = [], 0.0
    for b in range(0, n, 10):
        h = x[b:b + 10, None].double()
        for i, w in enumerate(ws):
            k = w.reshape(3, 3, 3, w.shape[1], w.shape[2]).permute(4, 3, 0, 1, 2)
            h = conv(h, k, padding=1)
            h = torch.relu(h) if i < 3 else h
        part = (m[b:b + 10].double() * (h[:, 0] - t[b:b + 10].double()) ** 2).sum() / m.double().sum()
        part.backward()
        loss_ref += float(part.detach())
        y_ref.append(h[:, 0].detach())
    y = torch.zeros_like(x)
    net.forward(x.data_ptr(), n, y.data_ptr())
    assert rel(y.cpu().numpy(), torch.cat(y_ref).cpu().numpy()) < 1e-2
    loss, gs = net.gradients(x.data_ptr(), t.data_ptr(), m.data_ptr(), n)
    assert abs(loss - loss_ref) <= 1e-2 * loss_ref
    for gr, w in zip(gs, ws):
        r = w.grad.cpu().numpy().reshape(gr.shape)
        assert rel(gr, r) < 3e-2, rel(gr, r)
    net.close()


@pytest.mark.parametrize("cell", [(9, 8, 7), (0, 0, 0), (17, 17, 17), (2, 0, 17), (3, 17, 0)])
def test_infinite_input_reaches_the_output(cell, require_gpu):
    """An infinite input is an infinite activation where its own tap is the
    only positive one, and the positive layers after it spread it to the cells
    within three of it; the others stay finite."""
    import torch
    net = fac.CNN(max_batch=1)
    w1 = np.full((27, 16), -0.3, dtype=np.float32)
    w1[13] = 0.5
    net.set_weights([w1] + [np.full(s, 0.01, dtype=np.float32) for s in fac.CNN_SHAPES[1:]])
    x = np.random.default_rng(3).random((1, S, S, S)).astype(np.float32)
    x[(0,) + cell] = np.inf
    xd = torch.from_numpy(x).cuda()
    y = torch.zeros_like(xd)
    net.forward(xd.data_ptr(), 1, y.data_ptr())
    far = np.abs(np.indices((S, S, S)) - np.reshape(cell, (3, 1, 1, 1))).max(axis=0)
    out = y.cpu().numpy()[0]
    assert np.array_equal(out == np.inf, far <= 3)
    assert np.isfinite(out[far > 3]).all()
    net.close()


def test_largest_output_gradients_stay_finite(require_gpu):
    """An output gradient beyond the largest BF16 number (3.39e38), which is a
    sum of three of them: the gradients are those of a 2^-20 times smaller one,
    scaled (1e-5: the order of the blocks' FP32 sums)."""
    import torch
    net = fac.CNN(max_batch=1)
    net.set_weights([np.full(s, 1e-3, dtype=np.float32) for s in fac.CNN_SHAPES])
    xd = torch.rand((1, S, S, S), generator=torch.Generator().manual_seed(1)).cuda()
    md = torch.zeros_like(xd)
    md[0, 9, 8, 7] = 1.0
    gs = []
    for scale in (1.0, 2.0 ** -20):
        td = -1.7e38 * scale * md
        gs.append(net.gradients(xd.data_ptr(), td.data_ptr(), md.data_ptr(), 1)[1])
    for g, h in zip(*gs):
        assert np.isfinite(g).all() and np.abs(g).max() > 0
        assert np.allclose(g * 2.0 ** -20, h, rtol=1e-5, atol=1e-5 * np.abs(h).max())
    net.close()

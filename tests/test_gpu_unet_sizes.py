"""The network at sizes where the fused steps can go wrong: images whose padded
frame is wider and taller than what is returned, single tiles, batches; the
image out of the last convolution against the CUDA-core path, and the fused
backward's parameter gradients against PyTorch, with the bounds of test_gpu_unet.py."""
import numpy as np
import pytest

from test_gpu_unet import MIN_COS, REL_L2, cosine, guides, perturbed, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (7, 9), (8, 8), (33, 17), (130, 71)])
def test_denoise_sizes(built, w, h):
    import torch
    from photon_tracer_b200.unet import UNet
    gen = torch.Generator(device="cuda").manual_seed(w * 100 + h)
    color, aux, depth = (torch.rand((h, w) + s, device="cuda", generator=gen) for s in ((3,), (7,), ()))
    net = UNet(seed=3)
    a = net.denoise(color, aux, depth)
    net.tensor_cores(False)
    b = net.denoise(color, aux, depth)
    net.sync()
    assert torch.isfinite(a).all() and float((a - b).norm() / b.norm()) < 1.5e-2  # as smoke() bounds it


@pytest.mark.parametrize("B,H,W", [(1, 24, 40), (3, 16, 72), (1, 136, 16)])
def test_gradients_at_sizes(built, B, H, W):
    import torch
    import unet_torch_ref as ref
    from photon_tracer_b200.unet import UNet, param_layout
    rng = np.random.default_rng(B * 1000 + H)
    x, target = guides(rng, B, H, W), np.full((B, H, W, 3), 1e4, np.float32)
    net = UNet(seed=5)
    p = perturbed(net, rng)
    loss, g, _ = net.loss_grads(torch.tensor(x, device="cuda"), torch.tensor(target, device="cuda"))
    r_loss, r_g, _, _ = ref.loss_and_grads(p, x, target)
    assert abs(loss - r_loss) <= 1e-3 * r_loss
    for i, (w_off, shape, b_off, co) in enumerate(param_layout()[0]):
        real = 3 if i == 14 else co  # only the 3 real outputs of the last layer get gradients
        n = int(np.prod(shape)) // co * real
        for off, count in ((w_off, n), (b_off, real)):
            assert rel_l2(g[off:off + count], r_g[off:off + count]) <= REL_L2, f"layer {i}"
            assert cosine(g[off:off + count], r_g[off:off + count]) >= MIN_COS, f"layer {i}"

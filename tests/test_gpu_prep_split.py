"""The fused preparation of few FP32 images of side 320 and 384, whose images several CTAs share: bit for
bit the values of a call of more images than are shared so (one CTA per image), and the oracle's
(relative L2 <= 1e-5, the bar of the preparation tests).  One image, the last number of images that is
split (37 on 148 SMs) and the first that is not; crops that leave some of the CTAs no rows; both
layouts; images off the 8-byte grid; two calls on the same scratch."""
import numpy as np
import pytest

import oracle
from frtest import rel_l2
from umpalumpa_b200.fr import Prep

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _cases(size):
    return [(0, 0, (1, 1, 1), None), (5, 6, (1, 1, 1), None), (size // 4 + 1, 34, (0, 1, 0), None),
            (size // 2, size - 2, (1, 0, 1), 0.06)]


@pytest.mark.parametrize("layout", ["rows", "banded"])
@pytest.mark.parametrize("size", [320, 384])
def test_split_images(cuda, size, layout):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    few = sms // 4
    imgs = np.random.default_rng(size).standard_normal((few + 1, size, size)).astype(np.float32)
    dev = torch.from_numpy(imgs).to(cuda)
    for out_x, out_y, flags, mf in _cases(size):
        p = Prep(size, size, out_x, out_y, *(bool(f) for f in flags), mf, layout=layout)

        def run(images):
            out = torch.zeros((images.shape[0], *p.out_shape), dtype=torch.complex64, device=cuda)
            got, _ = p.Execute(images, out)
            return got.data if layout == "banded" else got

        whole = run(dev)  # one CTA per image
        for n in (1, 2, few):
            assert torch.equal(run(dev[-n:]), whole[-n:]), (out_x, out_y, n)
        assert torch.equal(run(dev[:1]), whole[:1])
        if layout == "rows":
            ref = oracle.prepare_projections(imgs[-2:], out_x or None, out_y or None, *(bool(f) for f in flags), mf)
            assert rel_l2(whole[-2:].cpu().numpy(), ref) <= TOL


def test_split_images_off_the_8_byte_grid(cuda):
    import torch

    size = 320
    dev = torch.randn(3, size, size, device=cuda)
    flat = torch.zeros(dev.numel() + 1, dtype=torch.float32, device=cuda)
    flat[1:] = dev.flatten()
    shifted = flat[1:].view(dev.shape)
    assert shifted.data_ptr() % 8 == 4
    p = Prep(size, size)
    assert torch.equal(p.Execute(shifted)[0], p.Execute(dev)[0])


def test_small_calls_are_captured(cuda):
    import torch

    size = 384
    dev = torch.randn(2, size, size, device=cuda)
    st = torch.cuda.Stream()
    p = Prep(size, size, stream=st)
    out = torch.zeros((2, *p.out_shape), dtype=torch.complex64, device=cuda)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):  # the first call on the handle
        p.Execute(dev, out)
    for k in range(2):
        dev.normal_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, Prep(size, size).Execute(dev)[0])

"""The fused preparation at every side its FFT covers, against the oracle (relative L2 <= 1e-5, the
bar of the preparation tests): full and cropped half-planes (crops below one pass of 16 rows
and between two), a frequency crop, both layouts, one image and more images than CTAs, images at an
address that is not a multiple of 8, and 16-bit output equal to the quantised FP32 output."""
import numpy as np
import pytest

import oracle
from frtest import rel_l2
from umpalumpa_b200.fr import Prep, band_projections, quantize_projections

pytestmark = pytest.mark.gpu
TOL = 1e-5
SIDES = [64, 96, 128, 192, 256, 320, 384]


def _images(cuda, n, size):
    import torch

    imgs = np.random.default_rng(size).standard_normal((n, size, size)).astype(np.float32)
    return imgs, torch.from_numpy(imgs).to(cuda)


@pytest.mark.parametrize("size", SIDES)
def test_crops_and_flags(cuda, size):
    imgs, dev = _images(cuda, 3, size)
    for out_x, out_y, flags, mf in ((0, 0, (1, 1, 1), None), (5, 6, (1, 1, 1), None), (size // 4 + 1, size // 2 + 2, (0, 1, 0), None),
                                    (size // 2, size, (1, 0, 1), 0.06), (0, 0, (0, 0, 0), 0.2)):
        n, c, s = (bool(f) for f in flags)
        got, _ = Prep(size, size, out_x, out_y, n, c, s, mf, fft="fused").Execute(dev)
        ref = oracle.prepare_projections(imgs, out_x or None, out_y or None, n, c, s, mf)
        g = got.cpu().numpy()
        assert g.shape == ref.shape and rel_l2(g, ref) <= TOL, (out_x, out_y, rel_l2(g, ref))
        if mf:
            assert np.array_equal(g == 0, ref == 0)


@pytest.mark.parametrize("size", SIDES)
@pytest.mark.parametrize("storage", [0, 1, 2])
def test_layouts_and_storage(cuda, size, storage):
    import torch

    imgs, dev = _images(cuda, 950 if size == 64 else 2, size)  # side 64: more images than CTAs
    f32, _ = Prep(size, size, fft="fused").Execute(dev)
    rows, scales = Prep(size, size, storage=storage, fft="fused").Execute(dev)
    want, want_scales = (f32, None) if storage == 0 else quantize_projections(f32, storage)
    assert torch.equal(rows, want) and (storage == 0 or torch.equal(scales, want_scales))
    out = torch.zeros(Prep(size, size, storage=storage, layout="banded").out_shape, dtype=rows.dtype, device=cuda)
    out = torch.zeros((dev.shape[0], *out.shape, *rows.shape[3:]), dtype=rows.dtype, device=cuda)
    banded, _ = Prep(size, size, storage=storage, fft="fused", layout="banded").Execute(dev, out)
    assert torch.equal(banded.data, band_projections(want, storage).data)
    ref = oracle.prepare_projections(imgs[-2:])
    assert rel_l2(f32[-2:].cpu().numpy(), ref) <= TOL


def test_images_off_the_8_byte_grid(cuda):
    import torch

    size = 96
    imgs, dev = _images(cuda, 4, size)
    flat = torch.zeros(dev.numel() + 1, dtype=torch.float32, device=cuda)
    flat[1:] = dev.flatten()
    shifted = flat[1:].view(dev.shape)
    assert shifted.data_ptr() % 8 == 4
    a, _ = Prep(size, size, fft="fused").Execute(shifted)
    b, _ = Prep(size, size, fft="fused").Execute(dev)
    assert torch.equal(a, b)

"""The fused preparation of few FP32 images of side 192 and 256, shared by several CTAs as those of side 320
and 384 are: bit for bit the values of a call of more images than are shared so, and the oracle's
(relative L2 <= 1e-5, the bar of the preparation tests).  One image, the last number of images that is
split (three and two CTAs per SM, four of them an image) and the first that is not; crops that leave some
of the CTAs no rows; both layouts."""
import numpy as np
import pytest

import oracle
from frtest import rel_l2
from umpalumpa_b200.fr import Prep

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.mark.parametrize("layout", ["rows", "banded"])
@pytest.mark.parametrize("size,ctas", [(192, 3), (256, 2)])
def test_split_images(cuda, size, ctas, layout):
    import torch

    few = torch.cuda.get_device_properties(0).multi_processor_count * ctas // 4
    imgs = np.random.default_rng(size).standard_normal((few + 1, size, size)).astype(np.float32)
    dev = torch.from_numpy(imgs).to(cuda)
    for out_x, out_y, flags, mf in [(0, 0, (1, 1, 1), None), (5, 6, (1, 1, 1), None),
                                    (size // 4 + 1, 34, (0, 1, 0), None), (size // 2, size - 2, (1, 0, 1), 0.06)]:
        p = Prep(size, size, out_x, out_y, *(bool(f) for f in flags), mf, layout=layout)

        def run(images):
            out = torch.zeros((images.shape[0], *p.out_shape), dtype=torch.complex64, device=cuda)
            got, _ = p.Execute(images, out)
            return got.data if layout == "banded" else got

        whole = run(dev)  # one CTA per image
        for n in (1, 2, few):
            assert torch.equal(run(dev[-n:]), whole[-n:]), (out_x, out_y, n)
        if layout == "rows":
            ref = oracle.prepare_projections(imgs[-2:], out_x or None, out_y or None, *(bool(f) for f in flags), mf)
            assert rel_l2(whole[-2:].cpu().numpy(), ref) <= TOL

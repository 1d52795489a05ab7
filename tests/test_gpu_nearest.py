"""Nearest-pixel insertion (kFast) against the oracle (relative L2 <= 1e-5, the bar of the parity
tests) over storage, accumulation and half-plane layout, single job and batch, at volumes whose
last bricks hold one row of voxels and with list lengths 0, 1 and more per warp."""
import numpy as np
import pytest

import oracle
from frtest import rel_l2
from umpalumpa_b200 import synthetic
from umpalumpa_b200.fr import (FRB200, FRBatch, InputData, OutputData, Settings, band_projections,
                               quantize_projections)

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.mark.parametrize("box,n", [(16, 1), (32, 2), (46, 130), (64, 900)])
@pytest.mark.parametrize("storage,kahan", [(0, 0), (0, 1), (1, 0), (2, 1)])
def test_nearest(cuda, box, n, storage, kahan):
    import torch

    v = box + 1
    fft, rots = synthetic.make_job(box, n, seed=box + n, snr=0.1)
    spaces = oracle.traverse_spaces(rots, box // 2, box, box, box, use_fast=True)
    dev, scales, used = torch.from_numpy(fft).to(cuda), None, fft
    if storage:
        dev, scales = quantize_projections(dev, storage)
        pairs = (dev.float() * scales[:, None, None, None]).cpu().numpy()
        used = np.ascontiguousarray(pairs[..., 0] + 1j * pairs[..., 1]).astype(np.complex64)
    ov, ow = np.zeros((v, v, v), np.complex64), np.zeros((v, v, v), np.float32)
    oracle.fr_execute(ov, ow, used, spaces, interpolation=0, type_=0)
    sp = torch.from_numpy(spaces.view(np.uint8).reshape(-1, 112).copy()).to(cuda)
    for layout in (0, 1, 2):
        s = Settings()
        s.SetStorage(storage)
        s.SetAccumulation(kahan)
        s.SetLayout(layout)
        payload = band_projections(dev, storage) if layout == 2 else dev
        vol = torch.zeros((v, v, v), dtype=torch.complex64, device=cuda)
        w = torch.zeros((v, v, v), dtype=torch.float32, device=cuda)
        inp = InputData(payload, vol, w, sp, None, scales)
        op = FRB200(0)
        assert op.Init(OutputData(vol, w), inp, s), op.last_error
        assert op.Execute(OutputData(vol, w), inp), op.last_error
        op.Synchronize()
        assert rel_l2(w.cpu().numpy(), ow) <= TOL and rel_l2(vol.cpu().numpy(), ov) <= TOL, layout
        if layout == 1:
            continue
        vol.zero_()
        w.zero_()
        torch.cuda.synchronize()
        b = FRBatch(0)
        assert b.Init(s, 1, n, v), b.last_error
        assert b.Execute([inp]), b.last_error
        b.Synchronize()
        assert rel_l2(w.cpu().numpy(), ow) <= TOL and rel_l2(vol.cpu().numpy(), ov) <= TOL, ("batch", layout)

"""Nearest-pixel calls under the default layout read the caller's rows in place at every size: no banded
copy is made (its memory would show in the handle's bytes), and the result is the oracle's (relative
L2 <= 1e-5, the bar of every parity test).  Blob calls keep their copy."""
import numpy as np
import pytest

import oracle
from frtest import rel_l2
from umpalumpa_b200 import synthetic
from umpalumpa_b200.fr import FRB200, InputData, OutputData, Settings

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.mark.parametrize("fast", [True, False])
@pytest.mark.parametrize("box,n", [(16, 3), (48, 300), (64, 900)])
def test_no_copy(cuda, box, n, fast):
    import torch

    v = box + 1
    fft, rots = synthetic.make_job(box, n, seed=box + n, snr=0.1)
    spaces = oracle.traverse_spaces(rots, box // 2, box, box, box, use_fast=fast)
    ov, ow = np.zeros((v, v, v), np.complex64), np.zeros((v, v, v), np.float32)
    oracle.fr_execute(ov, ow, fft, spaces, interpolation=0, type_=0 if fast else 1)
    s = Settings()
    s.SetType(Settings.Type.kFast if fast else Settings.Type.kPrecise)
    vol = torch.zeros((v, v, v), dtype=torch.complex64, device=cuda)
    w = torch.zeros((v, v, v), dtype=torch.float32, device=cuda)
    inp = InputData(torch.from_numpy(fft).to(cuda), vol, w,
                    torch.from_numpy(spaces.view(np.uint8).reshape(-1, 112).copy()).to(cuda))
    op = FRB200(0)
    assert op.Init(OutputData(vol, w), inp, s), op.last_error
    before = op.GetUsedBytes()
    assert op.Execute(OutputData(vol, w), inp), op.last_error
    op.Synchronize()
    assert (op.GetUsedBytes() > before) == (not fast)
    assert rel_l2(w.cpu().numpy(), ow) <= TOL and rel_l2(vol.cpu().numpy(), ov) <= TOL

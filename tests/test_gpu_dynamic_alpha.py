"""Dynamic interpolation's polynomial over its range of alpha (up to 15) and at the first alpha
beyond it, through the single-job, batched and no-alloc entry points' shared constants, against
the float-decision FP64 oracle (relative L2 <= 1e-5, the bar of the parity tests; the
polynomial itself is within 2e-7).  Below alpha 4 the weight at the blob's edge is no longer small
(0.8 of its peak at alpha 1), so one tap whose squared distance rounds to the other side of r^2 --
the engine's is fused, the reference's not -- weighs more than the bar (1.1e-4 at one of 80 random
rotations); there the projections are axis-aligned, with whole-numbered distances."""
import numpy as np
import pytest

import oracle
from frtest import rel_l2
from umpalumpa_b200 import synthetic
from umpalumpa_b200.fr import FRB200, FRBatch, InputData, OutputData, Settings

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.mark.parametrize("alpha", [0.25, 1.0, 4.0, 7.5, 12.0, 15.0, 15.001])
@pytest.mark.parametrize("radius", [1.1, 1.9, 2.6])
def test_alpha_range(cuda, alpha, radius):
    import torch

    box, n = 32, 80
    v = box + 1
    fft, rots = synthetic.make_job(box, n, seed=int(10 * alpha), snr=0.1)
    if alpha < 4:
        eye = np.eye(3, dtype=np.float32)
        rots = np.stack([eye[[k % 3, (k + 1) % 3, (k + 2) % 3]] for k in range(n)]).astype(np.float32)
    spaces = oracle.traverse_spaces(rots, box // 2, box, box, box, radius=radius)
    dv, dw = oracle.fr_execute_fd64((v, v, v), fft, spaces, interpolation=0, type_=1, alpha=alpha, radius=radius)
    s = Settings()
    s.SetType(Settings.Type.kPrecise)
    s.SetAlpha(alpha)
    s.SetBlobRadius(radius)
    vol = torch.zeros((v, v, v), dtype=torch.complex64, device=cuda)
    w = torch.zeros((v, v, v), dtype=torch.float32, device=cuda)
    inp = InputData(torch.from_numpy(fft).to(cuda), vol, w,
                    torch.from_numpy(spaces.view(np.uint8).reshape(-1, 112).copy()).to(cuda))
    op = FRB200(0)
    assert op.Init(OutputData(vol, w), inp, s), op.last_error
    assert op.Execute(OutputData(vol, w), inp), op.last_error
    op.Synchronize()
    assert rel_l2(vol.cpu().numpy(), dv) <= TOL and rel_l2(w.cpu().numpy(), dw) <= TOL
    vol.zero_()
    w.zero_()
    torch.cuda.synchronize()
    b = FRBatch(0)
    assert b.Init(s, 1, n, v), b.last_error
    assert b.Execute([inp]), b.last_error
    b.Synchronize()
    assert rel_l2(vol.cpu().numpy(), dv) <= TOL and rel_l2(w.cpu().numpy(), dw) <= TOL

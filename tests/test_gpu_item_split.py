"""Work items of calls with few spaces: under the default item capacity the plan cuts the brick
lists shorter than 512 entries so that every brick group gets work; the result is the oracle's
(relative L2 <= 1e-5 on the volume and the weights, the bar of every parity test)."""
import numpy as np
import pytest

import oracle
from frtest import rel_l2
from umpalumpa_b200 import synthetic
from umpalumpa_b200.fr import FRB200, InputData, OutputData, Settings

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.mark.parametrize("kahan", [False, True])
@pytest.mark.parametrize("box,n", [(16, 1), (32, 3), (32, 64), (64, 1500)])
def test_short_items_match_oracle(cuda, box, n, kahan):
    import torch

    fft, rots = synthetic.make_job(box, n, seed=300 + box + n, snr=0.1)
    spaces = oracle.traverse_spaces(rots, box // 2, box, box, box)
    v = box + 1
    ov, ow = np.zeros((v, v, v), np.complex64), np.zeros((v, v, v), np.float32)
    oracle.fr_execute(ov, ow, fft, spaces, table=oracle.fill_blob_table())
    s = Settings()
    s.SetType(Settings.Type.kPrecise)
    s.SetInterpolation(Settings.Interpolation.kLookup)
    s.SetAccumulation(Settings.Accumulation.kKahan if kahan else Settings.Accumulation.kPlain)
    vol = torch.zeros((v, v, v), dtype=torch.complex64, device=cuda)
    w = torch.zeros((v, v, v), dtype=torch.float32, device=cuda)
    inp = InputData(torch.from_numpy(fft).to(cuda), vol, w,
                    torch.from_numpy(spaces.view(np.uint8).reshape(-1, 112).copy()).to(cuda),
                    torch.from_numpy(oracle.fill_blob_table()).to(cuda))
    op = FRB200(0)
    assert op.Init(OutputData(vol, w), inp, s), op.last_error
    items = {}
    for capacity in (512, 511):  # the default, cut as needed; any other capacity is taken as given
        op.set_launch_params(item_capacity=capacity)
        vol.zero_()
        w.zero_()
        assert op.Execute(OutputData(vol, w), inp), op.last_error
        op.Synchronize()
        assert rel_l2(w.cpu().numpy(), ow) <= TOL and rel_l2(vol.cpu().numpy(), ov) <= TOL
        items[capacity] = op.exec_stats().items
    bricks = ((v + 15) // 16) ** 3
    assert items[511] <= bricks * ((n + 510) // 511)
    if n >= 64:
        assert items[512] > items[511]
    if kahan:
        assert items[512] <= bricks * 8

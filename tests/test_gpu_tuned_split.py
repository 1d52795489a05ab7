"""A capacity from a tuning file is an upper bound, as the default is: a call of few spaces on a tuned
handle is cut into short items too.  One that the caller sets is taken as given, also after tuning.
Results are the oracle's (relative L2 <= 1e-5, the bar of every parity test)."""
import numpy as np
import pytest

import oracle
from frtest import rel_l2
from umpalumpa_b200 import _lib, synthetic
from umpalumpa_b200.fr import FRB200, FRBatch, InputData, OutputData, Settings

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _write(op, capacity, groups):
    key, path = op.TuningKey()
    with open(path, "w") as f:
        f.write(f"key={key}\ngroups={groups}\nctas_per_sm=1\nitem_capacity={capacity}\n")


@pytest.mark.parametrize("batch", [False, True])
@pytest.mark.parametrize("capacity", [128, 256, 512, 1024])
@pytest.mark.parametrize("kahan", [False, True])
def test_tuned_capacity_is_an_upper_bound(cuda, tmp_path, capacity, kahan, batch):
    import torch

    box, n = 32, 100
    v, groups = box + 1, 2 if kahan else 3
    fft, rots = synthetic.make_job(box, n, seed=5, snr=0.1)
    spaces = oracle.traverse_spaces(rots, box // 2, box, box, box)
    ov, ow = np.zeros((v, v, v), np.complex64), np.zeros((v, v, v), np.float32)
    oracle.fr_execute(ov, ow, fft, spaces, table=oracle.fill_blob_table())
    s = Settings()
    s.SetType(Settings.Type.kPrecise)
    s.SetInterpolation(Settings.Interpolation.kLookup)
    s.SetAccumulation(Settings.Accumulation.kKahan if kahan else Settings.Accumulation.kPlain)
    vol = torch.zeros((v, v, v), dtype=torch.complex64, device=cuda)
    w = torch.zeros((v, v, v), dtype=torch.float32, device=cuda)
    table = torch.from_numpy(oracle.fill_blob_table()).to(cuda)
    inp = InputData(torch.from_numpy(fft).to(cuda), vol, w,
                    torch.from_numpy(spaces.view(np.uint8).reshape(-1, 112).copy()).to(cuda), table)

    def init(op):
        if batch:
            assert op.Init(s, 1, n, v), op.last_error
        else:
            assert op.Init(OutputData(vol, w), inp, s), op.last_error

    def items(op):
        vol.zero_()
        w.zero_()
        torch.cuda.synchronize()
        done = op.Execute([inp], table) if batch else op.Execute(OutputData(vol, w), inp)
        assert done, op.last_error
        op.Synchronize()
        assert rel_l2(w.cpu().numpy(), ow) <= TOL and rel_l2(vol.cpu().numpy(), ov) <= TOL
        return op.exec_stats().items

    op = FRBatch(0) if batch else FRB200(0)
    init(op)
    op.SetTuning(_lib.FR_TUNING_CACHED, str(tmp_path))
    _write(op, capacity, groups)
    init(op)
    assert op.launch_params().item_capacity == capacity
    bricks = ((v + 15) // 16) ** 3
    assert items(op) > bricks  # 27 lists of at most 100 entries
    if batch:  # has no call to set them
        return
    op.set_launch_params(item_capacity=300)
    assert items(op) <= bricks
    op.set_launch_params(groups=1)  # the capacity stays the caller's
    assert items(op) <= bricks

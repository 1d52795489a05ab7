"""Launch parameters that the caller sets on a handle tuned from a file hold (the other fields stay the
file's); the handle stays tuned, so FR_TUNING_ON_EXECUTE starts no search for it."""
import os

import numpy as np
import pytest

import oracle
from umpalumpa_b200 import _lib, synthetic
from umpalumpa_b200.fr import FRB200, InputData, OutputData, Settings

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("approach", [_lib.FR_TUNING_CACHED, _lib.FR_TUNING_ON_EXECUTE])
def test_set_parameters_hold(cuda, tmp_path, approach):
    import torch

    box, n = 32, 20
    v = box + 1
    fft, rots = synthetic.make_job(box, n, seed=4, snr=0.1)
    spaces = oracle.traverse_spaces(rots, box // 2, box, box, box)
    vol = torch.zeros((v, v, v), dtype=torch.complex64, device=cuda)
    w = torch.zeros((v, v, v), dtype=torch.float32, device=cuda)
    inp = InputData(torch.from_numpy(fft).to(cuda), vol, w,
                    torch.from_numpy(spaces.view(np.uint8).reshape(-1, 112).copy()).to(cuda))
    s = Settings()
    s.SetType(Settings.Type.kPrecise)
    op = FRB200(0)
    assert op.Init(OutputData(vol, w), inp, s), op.last_error
    op.SetTuning(approach, str(tmp_path))
    key, path = op.TuningKey()
    text = f"key={key}\ngroups=2\nctas_per_sm=1\nitem_capacity=128\n"
    with open(path, "w") as f:
        f.write(text)
    assert op.Init(OutputData(vol, w), inp, s), op.last_error
    for change, want in (({"item_capacity": 300}, (2, 300)), ({"groups": 1}, (1, 300)), ({"item_capacity": 64}, (1, 64))):
        op.set_launch_params(**change)
        p = op.launch_params()
        assert (p.groups, p.item_capacity) == want
    assert op.Execute(OutputData(vol, w), inp), op.last_error
    op.Synchronize()
    p = op.launch_params()
    assert (p.groups, p.item_capacity) == (1, 64)
    assert open(path).read() == text and os.listdir(tmp_path) == [os.path.basename(path)]  # no search

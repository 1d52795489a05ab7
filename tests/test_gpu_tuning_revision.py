"""Tuning files written before the insertion kernels were changed (their key names no kernel revision)
are not taken: the shape they hold was the best of other kernels."""
import re

import numpy as np
import pytest

import oracle
from umpalumpa_b200 import _lib, synthetic
from umpalumpa_b200.fr import FRB200, FRBatch, InputData, OutputData, Settings

pytestmark = pytest.mark.gpu


def _fnv1a(text):
    h = 1469598103934665603
    for c in text.encode():
        h = ((h ^ c) * 1099511628211) % 2**64
    return h


@pytest.mark.parametrize("batch", [False, True])
def test_files_of_older_kernels_are_left_alone(cuda, tmp_path, batch):
    import torch

    box, n = 16, 4
    v = box + 1
    fft, rots = synthetic.make_job(box, n, seed=4, snr=0.1)
    spaces = oracle.traverse_spaces(rots, box // 2, box, box, box)
    vol = torch.zeros((v, v, v), dtype=torch.complex64, device=cuda)
    w = torch.zeros((v, v, v), dtype=torch.float32, device=cuda)
    inp = InputData(torch.from_numpy(fft).to(cuda), vol, w,
                    torch.from_numpy(spaces.view(np.uint8).reshape(-1, 112).copy()).to(cuda))
    s = Settings()
    s.SetType(Settings.Type.kPrecise)
    op = FRBatch(0) if batch else FRB200(0)

    def shape():
        assert op.Init(s, 1, n, v) if batch else op.Init(OutputData(vol, w), inp, s), op.last_error
        p = op.launch_params()
        return p.groups, p.item_capacity

    def write(key, path):
        with open(path, "w") as f:
            f.write(f"key={key}\ngroups=2\nctas_per_sm=1\nitem_capacity=128\n")

    op.SetTuning(_lib.FR_TUNING_CACHED, str(tmp_path))
    assert shape() == (3, 512)
    key, path = op.TuningKey()
    assert path.endswith("fr-b200-%016x.tune" % _fnv1a(key))
    old = re.sub(r" kernels=\d+", "", key)
    write(old, str(tmp_path / ("fr-b200-%016x.tune" % _fnv1a(old))))
    assert shape() == (3, 512)
    write(key, path)
    assert shape() == (2, 128)

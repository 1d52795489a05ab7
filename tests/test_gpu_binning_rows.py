"""The binning of brick rows at its edges, against the oracle (relative L2 <= 1e-5, the bar of the
parity tests): rows longer than the 32 bricks one CTA takes (a volume side above 512), volumes that
are not cubes of bricks, space counts around the 256 of a tile, and traverse spaces at an address
that is not a multiple of 16."""
import numpy as np
import pytest

import oracle
from frtest import rel_l2
from umpalumpa_b200 import synthetic
from umpalumpa_b200.fr import FRB200, FRBatch, InputData, OutputData, Settings

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _settings():
    s = Settings()
    s.SetType(Settings.Type.kPrecise)
    s.SetInterpolation(Settings.Interpolation.kLookup)
    return s


@pytest.mark.parametrize("box,n,offset", [(30, 255, 0), (32, 256, 4), (32, 257, 8), (46, 513, 12), (560, 2, 0)])
def test_rows(cuda, box, n, offset):
    import torch

    v = box + 1
    fft, rots = synthetic.make_job(box, n, seed=box + n, snr=0.1)
    spaces = oracle.traverse_spaces(rots, box // 2, box, box, box)
    table = oracle.fill_blob_table()
    ov, ow = np.zeros((v, v, v), np.complex64), np.zeros((v, v, v), np.float32)
    oracle.fr_execute(ov, ow, fft, spaces, table=table)
    raw = torch.zeros(n * 112 + 16, dtype=torch.uint8, device=cuda)
    sp = raw[offset:offset + n * 112].view(n, 112)
    sp.copy_(torch.from_numpy(spaces.view(np.uint8).reshape(-1, 112).copy()))
    assert sp.data_ptr() % 16 == offset
    vol = torch.zeros((v, v, v), dtype=torch.complex64, device=cuda)
    w = torch.zeros((v, v, v), dtype=torch.float32, device=cuda)
    tab = torch.from_numpy(table).to(cuda)
    inp = InputData(torch.from_numpy(fft).to(cuda), vol, w, sp, tab)
    op = FRB200(0)
    assert op.Init(OutputData(vol, w), inp, _settings()), op.last_error
    for calls in (1, 2):  # a second call starts its statistics anew
        vol.zero_()
        w.zero_()
        assert op.Execute(OutputData(vol, w), inp), op.last_error
        op.Synchronize()
        assert rel_l2(w.cpu().numpy(), ow) <= TOL and rel_l2(vol.cpu().numpy(), ov) <= TOL
        st = op.exec_stats()
        assert st.chunks == 1
        pairs = st.pairs if calls == 1 else pairs
        assert st.pairs == pairs
    vol.zero_()
    w.zero_()
    torch.cuda.synchronize()
    b = FRBatch(0)
    assert b.Init(_settings(), 1, n, v), b.last_error
    assert b.Execute([inp], tab), b.last_error
    b.Synchronize()
    assert b.exec_stats().pairs == pairs
    assert rel_l2(w.cpu().numpy(), ow) <= TOL and rel_l2(vol.cpu().numpy(), ov) <= TOL

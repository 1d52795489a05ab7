"""Voxels of the frequency sphere that map beyond the half-plane's far edges (half-planes cropped
below the sphere): no pixel lies within their blob, so they receive nothing -- whatever the space's
weight or the projection's scale, also where these are infinite or NaN."""
import numpy as np
import pytest

import oracle
from frtest import rel_l2
from umpalumpa_b200 import synthetic
from umpalumpa_b200.fr import FRB200, FRBatch, InputData, OutputData, Settings

pytestmark = pytest.mark.gpu
TOL = 1e-5  # the bar of the parity tests


def _job(cuda, box, n, fx, fy, storage=0, weight=1.0, scale=None):
    import torch

    v = box + 1
    fft, rots = synthetic.make_job(box, n, seed=5, snr=0.1)
    fft = np.ascontiguousarray(fft[:, :fy, :fx])
    spaces = oracle.traverse_spaces(rots, box // 2, box, box, box)
    spaces["weight"] = weight
    vol = torch.zeros((v, v, v), dtype=torch.complex64, device=cuda)
    w = torch.zeros((v, v, v), dtype=torch.float32, device=cuda)
    dev = torch.from_numpy(fft).to(cuda)
    scales = None
    if storage:
        dev = torch.view_as_real(dev).to(torch.bfloat16).contiguous()
        scales = torch.full((n,), scale, dtype=torch.float32, device=cuda)
    tab = torch.from_numpy(oracle.fill_blob_table()).to(cuda)
    sp = torch.from_numpy(spaces.view(np.uint8).reshape(-1, 112).copy()).to(cuda)
    return InputData(dev, vol, w, sp, tab, scales), fft, spaces


def _insert(inp, interp, layout, storage, batch):
    s = Settings()
    s.SetType(Settings.Type.kPrecise)
    s.SetInterpolation(interp)
    s.SetLayout(layout)
    s.SetStorage(storage)
    if interp == Settings.Interpolation.kDynamic:
        inp.blob_table = None
    out = OutputData(inp.volume, inp.weight)
    if batch:
        op = FRBatch(0)
        assert op.Init(s, 1, int(inp.traverse_space.shape[0]), int(inp.weight.shape[0])), op.last_error
        assert op.Execute([inp], inp.blob_table), op.last_error
    else:
        op = FRB200(0)
        assert op.Init(out, inp, s), op.last_error
        assert op.Execute(out, inp), op.last_error
    op.Synchronize()
    return inp.volume.cpu().numpy(), inp.weight.cpu().numpy()


@pytest.mark.parametrize("batch", [False, True])
@pytest.mark.parametrize("interp,layout", [(1, 0), (1, 1), (0, 0), (0, 1)])
@pytest.mark.parametrize("fx,fy", [(5, 8), (9, 16), (17, 16)])
def test_nothing_beyond_the_half_plane(cuda, fx, fy, interp, layout, batch):
    box, n = 32, 12
    inp, fft, spaces = _job(cuda, box, n, fx, fy)
    table = oracle.fill_blob_table() if interp else None
    ov, ow = np.zeros(inp.volume.shape, np.complex64), np.zeros(inp.weight.shape, np.float32)
    oracle.fr_execute(ov, ow, fft, spaces, table=table, interpolation=interp)
    gv, gw = _insert(inp, interp, layout, 0, batch)
    assert rel_l2(gv, ov) <= TOL and rel_l2(gw, ow) <= TOL
    hidden = _hidden(spaces, fx, fy, box)
    assert hidden.sum() > 100
    for storage, weight, scale in ((0, np.inf, None), (0, np.nan, None), (1, 1.0, np.inf)):
        inp, _, _ = _job(cuda, box, n, fx, fy, storage, weight, scale)
        gv, gw = _insert(inp, interp, layout, storage, batch)
        assert not np.isfinite(gv[ow > 0]).all()  # the voxels that see pixels do get it
        assert not gv[hidden].any() and not gw[hidden].any()


def _hidden(spaces, fx, fy, box, radius=1.9):
    """Voxels that lie beyond the half-plane's far edges, with a margin of 0.01, in every projection
    whose slab holds them (and in at least one)."""
    v = box + 1
    z, y, x = np.meshgrid(*[np.arange(v, dtype=np.float64) - box // 2] * 3, indexing="ij")
    p = np.stack([x, y, z])
    hidden, seen = np.zeros((v, v, v), bool), np.zeros((v, v, v), bool)
    for s in spaces:
        t = np.asarray(s["transformInv"], np.float64)
        q = np.einsum("ij,jzyx->izyx", t, p)
        slab = (np.abs(q[2]) <= radius + 0.01) & (q[0] >= -radius - 0.01)
        qy = q[1] + box // 2
        beyond = (q[0] > fx + radius + 0.01) | (qy < -radius - 0.01) | (qy > fy + radius + 0.01)
        hidden |= slab & beyond
        seen |= slab & ~beyond
    return hidden & ~seen

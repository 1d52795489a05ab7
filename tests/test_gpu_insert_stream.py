"""The insertion's voxel stream at its edges, against the oracle (relative L2 <= 1e-5, the bar of
every parity test): warps whose lists hold one voxel or none, blob radii whose columns are longer
than seven voxels (the list's second path), entries of more voxels than a warp's list takes (every column
of the brick visited whole), and spaces of different spheres and bounding boxes in one call."""
import numpy as np
import pytest

import oracle
from frtest import rel_l2
from umpalumpa_b200 import synthetic
from umpalumpa_b200.fr import FRB200, InputData, OutputData, Settings

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _run(cuda, box, fft, spaces, radius, layout=0, table=True):
    import torch

    v = box + 1
    s = Settings()
    s.SetType(Settings.Type.kPrecise)
    s.SetInterpolation(Settings.Interpolation.kLookup if table else Settings.Interpolation.kDynamic)
    s.SetBlobRadius(radius)
    s.SetLayout(layout)
    tab = oracle.fill_blob_table(radius=radius)
    vol = torch.zeros((v, v, v), dtype=torch.complex64, device=cuda)
    w = torch.zeros((v, v, v), dtype=torch.float32, device=cuda)
    inp = InputData(torch.from_numpy(fft).to(cuda), vol, w,
                    torch.from_numpy(spaces.view(np.uint8).reshape(-1, 112).copy()).to(cuda),
                    torch.from_numpy(tab).to(cuda) if table else None)
    op = FRB200(0)
    assert op.Init(OutputData(vol, w), inp, s), op.last_error
    assert op.Execute(OutputData(vol, w), inp), op.last_error
    op.Synchronize()
    ov, ow = np.zeros((v, v, v), np.complex64), np.zeros((v, v, v), np.float32)
    oracle.fr_execute(ov, ow, fft, spaces, table=tab if table else None, interpolation=int(table), radius=radius)
    return rel_l2(vol.cpu().numpy(), ov), rel_l2(w.cpu().numpy(), ow)


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("radius", [0.4, 1.0, 1.9, 2.4, 3.9])
def test_radii(cuda, radius, layout):
    box, n = 34, 45
    fft, rots = synthetic.make_job(box, n, seed=7, snr=0.1)
    spaces = oracle.traverse_spaces(rots, box // 2, box, box, box, radius=radius)
    assert max(_run(cuda, box, fft, spaces, radius, layout)) <= TOL


def test_mixed_spheres_boxes_and_weights(cuda):
    box, n = 40, 60
    fft, rots = synthetic.make_job(box, n, seed=8, snr=0.1)
    spaces = oracle.traverse_spaces(rots, box // 2, box, box, box)
    rng = np.random.default_rng(3)
    spaces["maxDistanceSqr"] *= rng.uniform(0.05, 1.0, n).astype(np.float32)
    spaces["weight"] = rng.uniform(0.5, 2.0, n).astype(np.float32)
    for lo, hi in (("minX", "maxX"), ("minY", "maxY"), ("minZ", "maxZ")):  # cut the traversal boxes
        spaces[lo] += rng.integers(0, 8, n).astype(np.int32)
        spaces[hi] -= rng.integers(0, 8, n).astype(np.int32)
    # The oracle walks the box on all three axes of a space's traversal, the engine leaves the
    # column axis open (the slab bounds it): keep that axis whole.
    for d, (lo, hi) in enumerate((("minZ", "maxZ"), ("minY", "maxY"), ("minX", "maxX"))):
        spaces[lo][spaces["dir"] == d] = 0
        spaces[hi][spaces["dir"] == d] = box
    assert max(_run(cuda, box, fft, spaces, 1.9)) <= TOL
    assert max(_run(cuda, box, fft, spaces, 1.9, table=False)) <= TOL


def test_axis_aligned_planes(cuda):
    """Planes along the bricks' faces: whole warps without a voxel beside warps whose 32 columns
    all hold the slab."""
    box = 32
    fft, _ = synthetic.make_job(box, 6, seed=9, snr=0.1)
    eye = np.eye(3, dtype=np.float32)
    rots = np.stack([eye, eye[[1, 2, 0]], eye[[2, 0, 1]], eye[[1, 2, 0]].T, -eye[[1, 0, 2]], eye[[0, 2, 1]] * [[1], [-1], [1]]])
    rots = np.ascontiguousarray(rots.astype(np.float32))
    spaces = oracle.traverse_spaces(rots, box // 2, box, box, box)
    assert max(_run(cuda, box, fft, spaces, 1.9)) <= TOL


@pytest.mark.parametrize("box,radius", [(4, 1.9), (6, 1.9), (10, 3.9)])
def test_half_planes_smaller_than_the_window(cuda, box, radius):
    n = 20
    fft, rots = synthetic.make_job(box, n, seed=box, snr=0.1)
    spaces = oracle.traverse_spaces(rots, box // 2, box, box, box, radius=radius)
    for layout in (0, 1):
        assert max(_run(cuda, box, fft, spaces, radius, layout)) <= TOL
        assert max(_run(cuda, box, fft, spaces, radius, layout, table=False)) <= TOL

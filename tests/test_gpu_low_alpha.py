"""Dynamic interpolation at low alpha over random rotations, through the single-job, batched and no-alloc
entry points, against the float-decision FP64 oracle (relative L2 <= 1e-5, the bar of the parity
tests).  Below alpha 4 the weight at the blob's edge is a sizeable part of the peak, so voxels with
a pixel within rounding distance of the radius -- the engine's squared distance is fused, the
reference's not, and either may count it -- are left out: |d^2 - r^2| < 4e-5, several times what FP32
leaves of d^2 = dx^2 + dy^2 + dz^2 <= r^2 at these coordinates (|q| <= 32: 2e-6 on each difference,
2 r 2e-6 on d^2).  They are few.

And the blob's polynomial itself over its whole range: weights from the engine's coefficients by FP32
Horner steps against I0 in FP64.  All 13 coefficients are rounded once and the steps once each, 25
roundings of at most 2^-24 of a sum of positive terms, 1.5e-6; the interpolation leaves less than
5e-7."""
import ctypes

import numpy as np
import pytest

import oracle
from frtest import rel_l2
from umpalumpa_b200 import _lib, synthetic
from umpalumpa_b200.fr import FRB200, FRBatch, InputData, OutputData, Settings, dims_of

TOL = 1e-5


def _off_the_edge(spaces, v, box, radius):
    """Voxels none of whose pixels lies within 4e-5 of r^2 (squared distance) in any projection."""
    keep = np.ones((v, v, v), bool)
    c = (v - 1) // 2
    z, y, x = np.meshgrid(*(np.arange(v) - c,) * 3, indexing="ij")
    p = np.stack([x, y, z], -1).astype(np.float64)
    for s in spaces:
        q = p @ np.asarray(s["transformInv"], np.float64).reshape(3, 3).T
        qx, qy, qz = q[..., 0], q[..., 1] + c, q[..., 2]
        near = (np.abs(qz) <= radius + 1e-3)
        fx, fy = np.floor(qx), np.floor(qy)
        for i in range(-3, 5):
            for j in range(-3, 5):
                d2 = (fx + i - qx) ** 2 + (fy + j - qy) ** 2 + qz**2
                keep &= ~(near & (np.abs(d2 - radius**2) < 4e-5))
    return keep


@pytest.mark.gpu
@pytest.mark.parametrize("alpha", [0.25, 1.0, 2.5, 3.9])
@pytest.mark.parametrize("radius", [1.1, 1.9, 2.6])
def test_low_alpha_random_rotations(cuda, alpha, radius):
    import torch

    box, n = 32, 24
    v = box + 1
    fft, rots = synthetic.make_job(box, n, seed=int(100 * alpha), snr=0.1)
    spaces = oracle.traverse_spaces(rots, box // 2, box, box, box, radius=radius)
    dv, dw = oracle.fr_execute_fd64((v, v, v), fft, spaces, interpolation=0, type_=1, alpha=alpha, radius=radius)
    keep = _off_the_edge(spaces, v, box, radius)
    touched = dw > 0
    assert keep[touched].mean() > 0.95
    s = Settings()
    s.SetType(Settings.Type.kPrecise)
    s.SetAlpha(alpha)
    s.SetBlobRadius(radius)
    vol = torch.zeros((v, v, v), dtype=torch.complex64, device=cuda)
    w = torch.zeros((v, v, v), dtype=torch.float32, device=cuda)
    inp = InputData(torch.from_numpy(fft).to(cuda), vol, w,
                    torch.from_numpy(spaces.view(np.uint8).reshape(-1, 112).copy()).to(cuda))

    def single():
        op = FRB200(0)
        assert op.Init(OutputData(vol, w), inp, s), op.last_error
        assert op.Execute(OutputData(vol, w), inp), op.last_error
        op.Synchronize()

    def batch():
        b = FRBatch(0)
        assert b.Init(s, 1, n, v), b.last_error
        assert b.Execute([inp]), b.last_error
        b.Synchronize()

    def noalloc():
        d, cs = dims_of(inp), s.to_c()
        rc = _lib.lib().fr_insert_noalloc(
            0, ctypes.c_void_p(torch.cuda.current_stream(0).cuda_stream), ctypes.byref(d), ctypes.byref(cs),
            ctypes.c_void_p(inp.fft.data_ptr()), None, n, ctypes.c_void_p(vol.data_ptr()), ctypes.c_void_p(w.data_ptr()),
            ctypes.c_void_p(inp.traverse_space.data_ptr()), n, None)
        assert rc == 0, _lib.last_error()

    for entry in (single, batch, noalloc):
        vol.zero_()
        w.zero_()
        torch.cuda.synchronize()
        entry()
        torch.cuda.synchronize()
        gv, gw = vol.cpu().numpy(), w.cpu().numpy()
        assert rel_l2(gv[keep], dv[keep]) <= TOL and rel_l2(gw[keep], dw[keep]) <= TOL, entry.__name__


@pytest.mark.parametrize("alpha", [0.01, 0.25, 1.0, 2.5, 4.0, 7.5, 10.0, 12.0, 15.0])
def test_polynomial_over_its_range(alpha):
    f = getattr(_lib.lib(), "_ZN3frb17kaiser_polynomialEffRA13_6float2")  # frb::kaiser_polynomial
    f.argtypes, f.restype = [ctypes.c_float, ctypes.c_float, ctypes.c_void_p], None
    c = np.zeros((13, 2), np.float32)
    f(alpha, 1.0, c.ctypes.data)
    assert np.array_equal(c[:, 0], c[:, 1])
    u = np.linspace(0.0, 1.0, 200001).astype(np.float32)
    h = np.full_like(u, c[12, 0])
    for k in range(11, -1, -1):  # fused: the product of two floats is exact in double
        h = (h.astype(np.float64) * u + np.float64(c[k, 0])).astype(np.float32)
    want = np.ones_like(u, np.float64)
    q, term = 0.25 * np.float64(np.float32(alpha)) ** 2 * u.astype(np.float64), np.ones_like(u, np.float64)
    for m in range(1, 60):
        term = term * q / (m * m)
        want = want + term
    assert np.max(np.abs(h - want) / want) <= 2e-6
    assert rel_l2(h, want) <= 3e-7

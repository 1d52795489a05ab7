"""Compensated sums of calls whose brick lists are cut for idle brick groups: merging a brick's
items may not cost accuracy, so the error against the float-decision FP64 oracle at the default
item capacity is that of one item per brick (capacity above every list, taken as given).

Both sums take the same terms and are compensated to 2^-8 of an FP32 rounding per add, so before
the last rounding they differ by a few percent of one rounding at these list lengths (at most
sqrt(400) 2^-8); the last rounding then falls differently in that share of the voxels.  Bar: 5 %.
Plain adds of the items gave 1.5 (lookup) and 2.7 times the error (nearest pixel) over eight calls."""
import ctypes

import numpy as np
import pytest

import oracle
from umpalumpa_b200 import _lib, synthetic
from umpalumpa_b200.fr import FRB200, FRBatch, InputData, OutputData, Settings, dims_of

pytestmark = pytest.mark.gpu


def _job(cuda, box, n, fast, lookup, seed):
    import torch

    fft, rots = synthetic.make_job(box, n, seed=seed, snr=0.1)
    spaces = oracle.traverse_spaces(rots, box // 2, box, box, box, use_fast=fast)
    table = oracle.fill_blob_table() if lookup else None
    v = box + 1
    s = Settings()
    s.SetType(Settings.Type.kFast if fast else Settings.Type.kPrecise)
    s.SetInterpolation(Settings.Interpolation.kLookup if lookup else Settings.Interpolation.kDynamic)
    s.SetAccumulation(Settings.Accumulation.kKahan)
    inp = InputData(torch.from_numpy(fft).to(cuda), torch.zeros((v, v, v), dtype=torch.complex64, device=cuda),
                    torch.zeros((v, v, v), dtype=torch.float32, device=cuda),
                    torch.from_numpy(spaces.view(np.uint8).reshape(-1, 112).copy()).to(cuda),
                    torch.from_numpy(table).to(cuda) if lookup else None)
    exact = oracle.fr_execute_fd64((v, v, v), fft, spaces, table=table, interpolation=int(lookup), type_=int(not fast))
    return inp, s, exact


def _errors(inp, exact):
    v, w = inp.volume.cpu().numpy(), inp.weight.cpu().numpy()
    return [float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel())) for a, b in zip((v, w), exact)]


def _part(inp, calls, k):
    n = inp.fft.shape[0]
    spaces = inp.traverse_space[n * k // calls:n * (k + 1) // calls].contiguous()
    return InputData(inp.fft, inp.volume, inp.weight, spaces, inp.blob_table)


def _insert(inp, s, calls, capacity, batch=False):
    inp.volume.zero_()
    inp.weight.zero_()
    out = OutputData(inp.volume, inp.weight)
    if batch:
        op = FRBatch(0)
        assert op.Init(s, 1, inp.fft.shape[0], inp.weight.shape[0]), op.last_error
    else:
        op = FRB200(0)
        assert op.Init(out, inp, s), op.last_error
        if capacity:
            op.set_launch_params(item_capacity=capacity)
    items = 0
    for k in range(calls):
        ok = op.Execute([_part(inp, calls, k)], inp.blob_table) if batch else op.Execute(out, _part(inp, calls, k))
        assert ok, op.last_error
        op.Synchronize()
        items += op.exec_stats().items
    return items


@pytest.mark.parametrize("calls", [1, 8])
@pytest.mark.parametrize("box,n,fast,lookup", [(32, 400, False, True), (32, 400, True, False), (48, 300, False, False),
                                               (64, 256, False, True)])
def test_cut_bricks_keep_the_accuracy(cuda, box, n, fast, lookup, calls):
    inp, s, exact = _job(cuda, box, n, fast, lookup, seed=1)
    whole = _insert(inp, s, calls, 511)
    ref = _errors(inp, exact)
    for batch in (False, True):
        items = _insert(inp, s, calls, 0, batch)
        got = _errors(inp, exact)
        assert items > whole or fast and calls == 8  # lists of fewer than 32 entries are not cut
        assert all(g <= 1.05 * r for g, r in zip(got, ref)), (batch, got, ref)


def test_sums_are_left_clear(cuda):
    """The sums' memory is zero again after a call, also where a brick was cut into the most items,
    and a call after it (other lists, other cut bricks) starts from zero."""
    import torch

    a, s, exact_a = _job(cuda, 64, 256, False, True, seed=1)
    b, _, exact_b = _job(cuda, 64, 256, False, True, seed=2)
    op = FRB200(0)
    assert op.Init(OutputData(a.volume, a.weight), a, s), op.last_error
    for _ in range(3):
        for inp, exact in ((a, exact_a), (b, exact_b)):
            inp.volume.zero_()
            inp.weight.zero_()
            assert op.Execute(OutputData(inp.volume, inp.weight), inp), op.last_error
            op.Synchronize()
            assert max(_errors(inp, exact)) <= 1e-6


# box 48: every brick's sums fit the fixed array; box 112: a third of them do
@pytest.mark.parametrize("box,n", [(48, 300), (112, 200)])
def test_no_alloc(cuda, box, n):
    import torch

    inp, s, exact = _job(cuda, box, n, False, True, seed=3)
    _insert(inp, s, 1, 511)
    ref = _errors(inp, exact)
    d, cs, st = dims_of(inp), s.to_c(), torch.cuda.current_stream(0)
    ptr = lambda t: None if t is None else ctypes.c_void_p(t.data_ptr())
    for _ in range(2):
        inp.volume.zero_()
        inp.weight.zero_()
        rc = _lib.lib().fr_insert_noalloc(0, ctypes.c_void_p(st.cuda_stream), ctypes.byref(d), ctypes.byref(cs),
                                          ptr(inp.fft), None, d.n_projections, ptr(inp.volume), ptr(inp.weight),
                                          ptr(inp.traverse_space), d.n_spaces, ptr(inp.blob_table))
        assert rc == 0, _lib.last_error()
        got = _errors(inp, exact)
        assert all(g <= 1.05 * r for g, r in zip(got, ref)), (got, ref)

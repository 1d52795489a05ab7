"""Launch parameters belong to the strategy they were resolved for: a handle initialised again for
another one starts from what its caller set, not from what the strategy before resolved to, and a
search's result applies to its own strategy alone."""
import numpy as np
import pytest

import oracle
from frtest import rel_l2
from umpalumpa_b200 import synthetic
from umpalumpa_b200.fr import FRB200, FRBatch, InputData, OutputData, Settings

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _settings(fast=False, kahan=False, storage=0):
    s = Settings()
    s.SetType(Settings.Type.kFast if fast else Settings.Type.kPrecise)
    s.SetAccumulation(Settings.Accumulation.kKahan if kahan else Settings.Accumulation.kPlain)
    s.SetStorage(storage)
    return s


def _job(cuda, box, n, fast=False):
    import torch

    v = box + 1
    fft, rots = synthetic.make_job(box, n, seed=11, snr=0.1)
    spaces = oracle.traverse_spaces(rots, box // 2, box, box, box, use_fast=fast)
    inp = InputData(torch.from_numpy(fft).to(cuda), torch.zeros((v, v, v), dtype=torch.complex64, device=cuda),
                    torch.zeros((v, v, v), dtype=torch.float32, device=cuda),
                    torch.from_numpy(spaces.view(np.uint8).reshape(-1, 112).copy()).to(cuda))
    return inp, fft, spaces


def _shape(op):
    p = op.launch_params()
    return p.groups, p.ctas_per_sm, p.item_capacity


# groups a CTA holds: three, two with compensations, one more without a blob table
STRATEGIES = {(False, False): 3, (False, True): 2, (True, False): 4, (True, True): 3}


@pytest.mark.parametrize("batch", [False, True])
def test_each_strategy_gets_its_own_defaults(cuda, batch):
    inp, _, _ = _job(cuda, 16, 4)
    op = FRBatch(0) if batch else FRB200(0)
    order = [(False, False), (True, False), (False, True), (False, False), (True, True), (True, False), (False, False)]
    for fast, kahan in order:
        s = _settings(fast, kahan)
        if batch:
            assert op.Init(s, 1, 4, 17), op.last_error
        else:
            assert op.Init(OutputData(inp.volume, inp.weight), inp, s), op.last_error
        assert _shape(op) == (STRATEGIES[fast, kahan], 1, 512), (fast, kahan)


def test_set_parameters_stay_set(cuda):
    inp, _, _ = _job(cuda, 16, 4)
    out = OutputData(inp.volume, inp.weight)
    op = FRB200(0)
    op.set_launch_params(item_capacity=300, groups=3)  # before the first Init
    assert op.Init(out, inp, _settings(kahan=True)), op.last_error
    assert _shape(op) == (2, 1, 300)  # three do not fit beside one another
    assert op.Init(out, inp, _settings()), op.last_error
    assert _shape(op) == (3, 1, 300)
    op.set_launch_params(groups=1)  # the other fields of this strategy stay
    assert _shape(op) == (1, 1, 300)
    op.set_launch_params(item_capacity=128)
    assert _shape(op) == (1, 1, 128)
    assert op.Init(out, inp, _settings(fast=True)), op.last_error
    assert _shape(op)[0] == 1 and _shape(op)[2] == 128


@pytest.mark.parametrize("groups", [1, 2, 3, 4])
@pytest.mark.parametrize("kahan", [False, True])
def test_nearest_pixel_shapes(cuda, groups, kahan):
    inp, fft, spaces = _job(cuda, 48, 300, fast=True)
    ov, ow = np.zeros(inp.volume.shape, np.complex64), np.zeros(inp.weight.shape, np.float32)
    oracle.fr_execute(ov, ow, fft, spaces, interpolation=0, type_=0)
    op = FRB200(0)
    assert op.Init(OutputData(inp.volume, inp.weight), inp, _settings(True, kahan)), op.last_error
    op.set_launch_params(item_capacity=128, groups=groups)
    assert _shape(op)[0] == min(groups, STRATEGIES[True, kahan])
    assert op.Execute(OutputData(inp.volume, inp.weight), inp), op.last_error
    op.Synchronize()
    assert rel_l2(inp.volume.cpu().numpy(), ov) <= TOL and rel_l2(inp.weight.cpu().numpy(), ow) <= TOL


def test_a_search_applies_to_its_strategy(cuda):
    inp, _, _ = _job(cuda, 48, 600)
    out = OutputData(inp.volume, inp.weight)
    op = FRB200(0)
    assert op.Init(out, inp, _settings()), op.last_error
    op.Autotune(inp)
    tuned = _shape(op)
    assert op.Init(out, inp, _settings(fast=True)), op.last_error
    assert _shape(op) == (4, 1, 512)
    assert op.Init(out, inp, _settings()), op.last_error
    assert _shape(op) == tuned

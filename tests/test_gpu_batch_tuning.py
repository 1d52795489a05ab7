"""A batched handle takes the launch parameters of its strategy's tuning file: at Init under
FR_TUNING_CACHED, and when that approach is set after Init; a file of another strategy (other
limits) is left alone."""
import pytest

from umpalumpa_b200 import _lib
from umpalumpa_b200.fr import FRBatch, Settings

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("after", [False, True])
def test_a_batch_takes_its_tuning_file(cuda, tmp_path, after):
    s = Settings()
    s.SetType(Settings.Type.kPrecise)
    b = FRBatch(0)
    assert b.Init(s, 2, 100, 33), b.last_error
    b.SetTuning(_lib.FR_TUNING_CACHED, str(tmp_path))
    key, path = b.TuningKey()
    with open(path, "w") as f:
        f.write(f"key={key}\ngroups=2\nctas_per_sm=1\nitem_capacity=128\n")
    c = FRBatch(0)
    if not after:
        c.SetTuning(_lib.FR_TUNING_CACHED, str(tmp_path))
    assert c.Init(s, 2, 100, 33), c.last_error
    if after:
        c.SetTuning(_lib.FR_TUNING_CACHED, str(tmp_path))
    p = c.launch_params()
    assert (p.groups, p.item_capacity) == (2, 128)
    assert c.Init(s, 3, 100, 33), c.last_error
    p = c.launch_params()
    assert (p.groups, p.item_capacity) == (3, 512)

"""The autotuner's cache: an entry applies to the forms it was timed against."""
import json

import pytest

from tfhe_b200 import autotune as A
from tfhe_b200.params import CONFIG1


class FakeKeys:
    params = CONFIG1

    def __init__(self, forms):
        self.forms, self.applied = forms, None

    def launches(self, batch):
        return [(batch, k, c) for k, c in self.forms]

    def launch_shape(self, batch):
        return 2, 256, 0

    def set_tuning(self, *shape):
        self.applied = shape


@pytest.fixture
def timed(monkeypatch):
    """Without a GPU: a name, no inputs, and (0, 0, 1) the fastest shape."""
    calls = []
    monkeypatch.setattr(A.torch.cuda, "get_device_name", lambda *_: "GPU")
    monkeypatch.setattr(A.torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(A.torch, "device", lambda *_: "cpu")
    monkeypatch.setattr(A, "time_shape", lambda keys, shape, *_: calls.append(shape) or (0.5 if shape == (0, 0, 1) else 1.0))
    return calls


def test_a_shape_of_other_forms_is_not_applied(tmp_path, timed):
    path = str(tmp_path / "tune.json")
    before = FakeKeys([(2, 1)])
    # the key of a library that knew no forms beside the shapes
    with open(path, "w") as fh:
        json.dump({f"GPU|{CONFIG1.name}|256": {"shape": [2, -1, 0]}}, fh)
    assert A.autotune(before, 256, path=path)[0] == (0, 0, 1) and timed
    timed.clear()
    assert A.autotune(before, 300, path=path) == ((0, 0, 1), {})     # the same forms: applied untimed
    assert not timed and before.applied == (0, 0, 1)
    after = FakeKeys([(4, 2)])
    assert A.autotune(after, 256, path=path)[1] and timed            # other forms: timed anew

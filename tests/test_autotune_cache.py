"""The autotuner's cache (CPU only): a winner is applied to the kernels it was timed on, and to no others."""
import json
import types

import numpy as np

from vamtoolbox_b200 import autotune

OLD = {"forward_vz": 1, "backward_vz": 4, "adjoint_vz": 1, "backward_batch": 2, "adjoint_table": 1,
       "backward_table": 0, "forward_tma": 1}


class Plan:
    shape_vol, angles, absorption, has_occlusion, device = (96, 96, 33), np.zeros(90), None, False, None

    def __init__(self):
        self.tuning = {}

    def set_tuning(self, t):
        self.tuning = dict(t)

    def get_tuning(self):
        return self.tuning


def test_winners_of_other_kernels_are_not_applied(tmp_path, monkeypatch):
    """An entry keyed without a revision (as written before keys had one) or with another one is a miss: the shapes
    are timed again.  The entry then written is applied without timing."""
    path = tmp_path / "tuning.json"
    monkeypatch.setenv("VAMTOOLBOX_B200_TUNE_CACHE", str(path))
    monkeypatch.setattr(autotune, "torch", types.SimpleNamespace(
        cuda=types.SimpleNamespace(get_device_name=lambda device: "A GPU")))
    timed = []
    monkeypatch.setattr(autotune, "measure", lambda plan, *a: (timed.append(plan) or {"forward_vz": 4}, {}))
    shape = "A_GPU|96x96x33|na90|abs=none|occ=0"
    path.write_text(json.dumps({k: {"tuning": OLD, "ms": {}} for k in (shape, "k1|" + shape)}))
    assert autotune.autotune(Plan()) == {"forward_vz": 4} and len(timed) == 1
    assert autotune.autotune(Plan()) == {"forward_vz": 4} and len(timed) == 1
    assert shape in autotune.problem_key(Plan())

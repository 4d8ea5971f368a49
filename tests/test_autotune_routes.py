"""The tuner and the route of a call: a handle whose TD calls run on chip keeps kernel 0
(kernel 1 would switch the resident loop off), also from the cache; choices stored for
another set of kernels are measured anew."""
import json

import numpy as np

from svirl_gb300 import autotune as AT
from tests.test_autotune import FakeHandle


class OnChip(FakeHandle):
    def td_resident(self):
        return True


def test_resident_handles_keep_kernel_0(tmp_path):
    path = str(tmp_path / "tune.json")
    times = {(0, 12): 0.05, (1, 8): 0.01}
    away = FakeHandle(np.float32, times=times)
    assert AT.tune(away, path=path)["kernel"] == 1 and away.kernel == 1
    for force in (False, True):
        h = OnChip(np.float32, times=times)
        c = AT.tune(h, path=path, force=force)
        assert c["cached"] != force and c["kernel"] == 0 and h.kernel == 0
    assert c["rows"] == 12 and c["us"] == c["measured"]["0/12"]


def test_choices_of_other_kernels_are_not_taken(tmp_path):
    path = str(tmp_path / "tune.json")
    h = FakeHandle(np.float32, times={(0, 8): 0.02})
    old = "float32:%dx%d:finite" % (h.Nx, h.Ny)  # without the kernel set
    json.dump({old: {"kernel": 1, "rows": 17, "us": 1.0, "measured": {}}}, open(path, "w"))
    c = AT.tune(h, path=path)
    assert not c["cached"] and h.kernel == 0
    assert set(json.load(open(path))) == {old, AT.key_of(h)}

"""The autotuner's search, on the CPU: no two values of a parameter run the same code, and
winners cached for kernels that read a value otherwise are not taken."""
import json

import pytest

from smallproject_gb300 import autotune as at
from smallproject_gb300 import vxr as V


def _effect(name, value):
    """What the default tracer makes of a searched value."""
    if name == "shadow_burst":
        return -(-value // 4)                                 # rounds of 4 visits
    if name == "shadow_refill":
        return max(value >> 1, 1), max(value >> 2, 1)         # candidates, shading
    return value


@pytest.mark.parametrize("name, values", at.SPACE)
def test_searched_values_differ_in_effect(name, values):
    assert len({_effect(name, v) for v in values}) == len(values)
    default = at._from_tuning(V.tuning())[name]
    assert default in values


def test_winners_of_other_kernels_are_not_taken(monkeypatch, tmp_path):
    monkeypatch.setattr(V, "device_info", lambda: ("GPU", 152, (10, 3)))
    monkeypatch.setattr(at, "_world_class", lambda world: (6, 11))

    class View:
        desc = V.view_desc(640, 360, V.LIGHTS_POINT)
        took = None

        def set_tuning(self, t):
            self.took = t

    path = str(tmp_path / "cache.json")
    view = View()
    key = at.config_key(None, view.desc)
    winner = {"tuning": {"tile": [32, 4], "persistent": 0, "shadow_refill": 24, "shadow_burst": 8,
                         "list_blocks_per_sm": 8}, "ms": 1.0}
    # the generation before refill counts were split between the two passes, and none at all
    old = key.rsplit("|", 1)[0]
    with open(path, "w") as fh:
        json.dump({old: winner, old + "|split": winner}, fh)
    assert at.apply_cached(view, None, path) is False and view.took is None
    with open(path, "w") as fh:
        json.dump({key: winner}, fh)
    assert at.apply_cached(view, None, path) is True and view.took.shadow_refill == 24

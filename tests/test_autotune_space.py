"""The autotuner's search, on the CPU: no two values of a parameter run the same code."""
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

"""What kernels launched while the one before them still runs may touch
before they wait for it (engine/device.cuh, previous_done): run-constant
data only.  The writes of earlier kernels, also of those that have finished,
are visible only after the wait, and a read too early shows in no result
that can be relied on to repeat, so the sources are checked."""
import re

import pytest

from conftest import ROOT

CSRC = ROOT / "dust2_gb300" / "csrc"
FILES = ["filter_kernels.cu", "engine/filter.cuh", "engine/continuous.cuh",
         "engine/kernels_common.cuh"]
# written by the kernels of a filter's observation loop
WRITTEN = re.compile(
    r"\bf\.(w|ew|pre|idx|mode|ll|frng|gkey|gnz|gflag|gu|gtot|guu0|gdu|"
    r"chunk_sum|chunk_off)\b"
    r"|\bv\.(state|rng|errors|any_error)\b"
    r"|\b(draw_group_uniform|group_has_sum|scaled_weight|load_rng|load_state|"
    r"load_column|load_ode|load_ode_scalars|keep_tile|step_particle)\s*[(<]"
    r"|\b(src|dst|index|group_mode|state|idx|mode)\s*\[")


def waits():
    for name in FILES:
        text = (CSRC / name).read_text()
        for m in re.finditer(r"^ *previous_done\(\);", text, re.M):
            # the function's body so far, lambdas (called later) left out
            start = text.rfind("\n}\n", 0, m.start())
            body = text[start:m.start()]
            body = re.sub(r"//[^\n]*", "", body)
            body = re.sub(r"auto \w+ = \[[&=]?\][^{]*\{\n.*?\n  \};", "",
                          body, flags=re.S)
            yield name, text.count("\n", 0, m.start()) + 1, body


def test_every_kernel_is_found():
    assert len(list(waits())) >= 12


@pytest.mark.parametrize("where", list(waits()),
                         ids=lambda w: f"{w[0]}:{w[1]}")
def test_nothing_written_is_read_before_the_wait(where):
    found = WRITTEN.search(where[2])
    assert found is None, found.group(0)

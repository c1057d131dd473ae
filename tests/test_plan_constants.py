"""Numbers that the header and the Python side state alike."""

from __future__ import annotations

import re
from pathlib import Path

import pytest

from abstraction_regret_gb300 import native

HEADER = (Path(__file__).resolve().parent.parent / "include" / "gbfsm.h").read_text()


@pytest.mark.parametrize("name", ["PLAN_DFA_BALANCE", "DFA_RARE_ACCEPT", "DFA_COLLAPSES",
                                  "CODE_SET", "LANE_STAGE_WIDE", "LANE_STAGE_NARROW"])
def test_python_states_the_header_s_number(name):
    value = re.search(rf"#define GBFSM_{name} (\S.*?)(?:/\*|$)", HEADER, re.M).group(1)
    assert eval(value.replace("u", "")) == getattr(native, name)  # noqa: S307 - a constant

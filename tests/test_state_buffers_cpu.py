"""Every device buffer of the library's state is released with it and counted in its size."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cosmosphere_b200", "csrc")


def _buffers():
    with open(os.path.join(CSRC, "state.hpp")) as f:
        state = f.read().split("struct State\n")[1].split("\n};")[0]
    names = []
    for decl in re.findall(r"^\s*DBuf<\w+>\s+([^;]+);", state, flags=re.M):
        names += [re.sub(r"\[\d+\]", "", d).strip() for d in decl.split(",")]
    return names


@pytest.mark.parametrize("function", ["size_t state_device_bytes", "void release_state"])
def test_every_buffer_of_the_state(function):
    with open(os.path.join(CSRC, "c_api.cu")) as f:
        body = f.read().split("\n" + function)[1].split("\n}")[0]
    names = _buffers()
    assert len(names) > 80
    assert [n for n in names if not re.search(r"\bs\." + n + r"\b", body)] == []

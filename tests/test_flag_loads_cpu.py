"""Flags that a kernel reads behind a grid-dependency wait: the previous kernel in the stream may be the one
that writes them, and the compiler may move a read-only load (__ldg) above the wait, so the code that runs
there loads them by volatile statements."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "mojo_lbm_gb300" / "csrc"


def _body(file: str, name: str) -> str:
    """The text of the function `name` (from its definition to the closing brace in column 0)."""
    text = (CSRC / file).read_text()
    at = re.search(rf"\b{name}\([^;]*?\) \{{", text)
    assert at, name
    return text[at.start():text.index("\n}", at.start())]


@pytest.mark.parametrize("file,name", [("lbm_capi.cu", "load_flags16"), ("lbm_capi.cu", "tile_check_kernel"),
                                       ("lbm_capi.cu", "rebuild_tile"), ("lbm_step.cuh", "any_solid_masks"),
                                       ("lbm_step.cuh", "cell_solid_masks"), ("lbm_step.cuh", "step_kernel")])
def test_no_read_only_loads_of_flags(file, name):
    assert "__ldg" not in _body(file, name)

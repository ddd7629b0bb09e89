"""The teams of threads that share an element leave a kernel as a whole: a body with shuffles, reductions or barriers
over a team's mask reads the words that another stream may write meanwhile through a vote of the team alone. (A
thread that left by itself would be missing from them, which could hang the others, so this is read from the
source.)"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "edg_westervelt_gb300", "csrc")
FILES = ["wedg_kernels.cuh", "wedg_stage_fx.cuh", "wedg_stage_gen.cuh", "wedg_adjoint.cuh"]


def _bodies(text):
    """(name, source) of the device functions and of the macros that bodies begin with."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__device__ __forceinline__ [\w ]*?\b(\w+)\(([^;{]*)\)\s*(?:const )?{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m[1], text[m.end():i]
    for m in re.finditer(r"#define (\w+)(?:\([^)]*\))? \\\n((?:.*\\\n)*.*\n)", text):
        yield m[1], m[2]


@pytest.mark.parametrize("name", FILES)
def test_teams_leave_as_a_whole(name):
    with open(os.path.join(CSRC, name)) as f:
        bodies = dict(_bodies(f.read()))
    assert bodies
    macros = {k: v for k, v in bodies.items() if k.startswith("WEDG_")}
    teams = 0
    for fn, src in bodies.items():
        for m, v in macros.items():
            if fn != m and re.search(rf"\b{m}\b", src):
                src += v
        if "(mask" not in src:
            continue
        teams += 1
        for m in re.finditer(r"[^\n;]*\berr_word\(F\)[^\n]*|[^\n;]*\*\(volatile[^\n]*F\.err[^\n]*", src):
            line = m[0]
            assert "__any_sync(mask" in line or "return" not in line or fn == "prep_stopped", (fn, line.strip())
    assert teams >= 1

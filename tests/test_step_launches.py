"""Kernels launched with programmatic serialization start before the grid
ahead of them has ended, and only griddepcontrol.wait makes that grid's writes
visible to them: each must execute it in every thread, unconditionally."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "simlab_b200" / "csrc"
WAIT = r'(?:lbm::)?pdl_wait\(\);|asm volatile\("griddepcontrol\.wait;" ::: "memory"\);'


def _sources():
    return {f.name: f.read_text() for f in sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh"))}


def _launched():
    names = set()
    for text in _sources().values():
        names |= {m.split("::")[-1] for m in re.findall(r"launch_pdl\([^,()]+,\s*([\w:]+)\s*[<,]", text)}
        names |= {m.split("::")[-1] for m in re.findall(r"cudaLaunchKernelEx\(&cfg,\s*([\w:]+)\s*<", text)}
    return sorted(names)


def _body(name):
    for text in _sources().values():
        m = re.search(r"__global__[^;{]*\b" + name + r"\([^{;]*\)\s*\{\n(.*?)\n\}\n", text, re.S)
        if m:
            return m.group(1)
    return None


def test_there_are_such_kernels():
    assert {"k_faces", "k_walls", "k_bulk_tma", "k_voxelize", "k27_step", "k27_walls", "kg_step"} <= set(_launched())


@pytest.mark.parametrize("name", _launched())
def test_every_thread_waits_for_the_grid_ahead(name):
    body = _body(name)
    assert body is not None
    # a statement of the kernel's own block, not of a branch or a loop in it
    w = re.search(r"^    (?:" + WAIT + ")", body, re.M)
    assert w, "no unconditional wait"
    before = re.sub(r"//[^\n]*", "", body[: w.start()])
    # nothing of the step's state is read, and no thread leaves, ahead of it
    assert not re.search(r"\breturn\b|p\.(?:pop|flags|recs|recd|faces|mom|partials|sol|qscr)\b|\b(?:src|dst|lin|lout|mom)\[", before)

"""A kernel launched as a programmatic dependent may be resident while the
kernel before it still writes, so after its wait it reads through ordinary
loads or TMA, never through the read-only path (ld.global.nc is for data that
is not written while the kernel lives, and no wait orders it).  Checked on the
sources: no result shows a load of the wrong kind for certain."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "gpe_b200" / "csrc"


def code(path):
    """The source without its comments."""
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)


def waits():
    """(name, code after the wait) of every function that waits for the kernel before it."""
    out = []
    for path in sorted(CSRC.glob("*.cu*")):
        src = code(path)
        for m in re.finditer(r"pdl_wait\(\);", src):
            # functions end at a closing brace in the first column
            start, end = src.rfind("\n}", 0, m.start()), src.find("\n}", m.start())
            head = re.sub(r"\b(template|launch_bounds__|typename|sizeof)\b", "", src[start:m.start()])
            name = re.search(r"(\w+)\s*\((?:const )?(?:__grid_constant__ )?(?:const )?(?:TmaMaps|StageArgs)", head)
            out.append((f"{path.name}:{name.group(1) if name else '?'}", src[m.end():end]))
    return out


def test_the_waiting_kernels_are_found():
    names = {n for n, _ in waits()}
    assert {"gpe_device.cuh:k_stage_site", "gpe_stage_tma.cuh:tma_item", "gpe_stage_tma.cuh:tma_item_pair"} <= names


@pytest.mark.parametrize("name,body", waits(), ids=[n for n, _ in waits()])
def test_no_read_only_load_after_the_wait(name, body):
    assert not re.search(r"\bldro\s*\(|\b__ldg\w*\s*\(|ld\.global\.nc", body), name

"""Every kernel that is launched behind the one before it (launch_behind) waits
for that one on the device before it touches memory: read from the sources, as a
missing wait shows in no result while the kernel before happens to be done."""
import glob
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "n-body_gb300", "csrc")
WAIT = "wait_for_launches_before();"


def _sources():
    text = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        s = open(path).read()
        s = re.sub(r"/\*.*?\*/", "", s, flags=re.S)
        text[os.path.basename(path)] = re.sub(r"//[^\n]*", "", s)
    return text


def _closing(s, at, pair):
    depth = 0
    for i in range(at, len(s)):
        depth += (s[i] == pair[0]) - (s[i] == pair[1])
        if depth == 0:
            return i
    raise ValueError("unbalanced source")


def _kernels():
    """name -> (pointer parameters, body)"""
    found = {}
    for s in _sources().values():
        for m in re.finditer(r"__global__\s+void\s+", s):
            at = m.end()
            bounds = re.match(r"__launch_bounds__\s*\(", s[at:])
            if bounds:
                at = _closing(s, at + bounds.end() - 1, "()") + 1
            name = re.match(r"\s*(\w+)\s*\(", s[at:])
            first = at + name.end() - 1
            last = _closing(s, first, "()")
            body = s.index("{", last)
            pointers = re.findall(r"\*\s*(?:__restrict__\s+)?(\w+)\s*(?=[,)])", s[first:last + 1])
            found[name.group(1)] = (pointers, s[body:_closing(s, body, "{}") + 1])
    return found


def _launched_behind():
    names = set()
    for s in _sources().values():
        names.update(m for m in re.findall(r"launch_behind\s*\(\s*(\w+)", s) if m != "void")
        names.update(re.findall(r"\blaunch\s*\(\s*(\w+_kernel)\b", s))  # by way of a generic lambda
    return sorted(n for n in names if n.endswith("_kernel"))


KERNELS = _kernels()


def test_launches_are_found():
    names = _launched_behind()
    assert len(names) >= 25 and set(names) <= set(KERNELS)
    assert {"bbox_kernel", "seg_keys_kernel", "team_walk_kernel", "pp_sym_kernel", "merge_pass_kernel"} <= set(names)


@pytest.mark.parametrize("name", _launched_behind())
def test_kernel_waits_before_it_touches_memory(name):
    pointers, body = KERNELS[name]
    assert WAIT in body, f"{name} is launched behind the kernel before it and never waits for it"
    before = body[:body.index(WAIT)]
    touched = [p for p in pointers if re.search(rf"\b{p}\b", before)]
    if "kWalkWaitsLast" in before:  # begins beside the walk before it, by that walk's word
        assert "load_acquire(ready)" in before, f"{name} skips the wait without an acquire of what it reads"
        touched.remove("ready")
    else:
        assert body.count(WAIT) == 1
    assert not touched, f"{name} uses {touched} before it waits"


@pytest.mark.parametrize("name", ["cell_walk_kernel", "team_walk_kernel"])
def test_walk_says_that_it_has_waited_before_it_lets_the_next_begin(name):
    body = KERNELS[name][1]
    said, let = body.index("store_release(ready"), body.index("let_next_launch_begin();")
    assert body.index(WAIT) < said < let

"""Distributed shared memory in the cluster kernels, by their source: a CTA of a cluster may
touch another's shared memory only after a barrier that all CTAs of the cluster have
reached, since nothing else says that they have started."""

import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "pytential_b200", "csrc")


def _functions():
    """(name, body) of every function that maps another CTA's shared memory; a namespace's
    bodies are found by the braces that open at the start of a line."""
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for m in re.finditer(r"^\{\n(.*?)^\}", text, re.S | re.M):
            if "map_shared_rank" in m.group(1):
                name = re.findall(r"(\w+)\s*\(", text[:m.start()].rsplit("\n\n", 1)[-1])[-1]
                out.append((os.path.basename(path) + ":" + name, m.group(1)))
    return out


def test_all_uses_are_found():
    uses = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        with open(path) as f:
            uses += len(re.findall(r"map_shared_rank", re.sub(r"//[^\n]*", "", f.read())))
    assert uses == sum(b.count("map_shared_rank") for _, b in _functions()) > 0


@pytest.mark.parametrize("name,body", _functions(), ids=[n for n, _ in _functions()])
def test_barrier_before_first_remote_access(name, body):
    first = body.index("map_shared_rank")
    assert re.search(r"\bcl\.(sync|barrier_wait)\s*\(", body[:first]), \
        f"{name}: no cluster barrier before the first access to another CTA's shared memory"

"""Ordering that the kernels' sources have to state because no result shows its absence (csrc/orbit_pair.cuh)."""

import os
import re

import pytest
from conftest import ROOT

CSRC = os.path.join(ROOT, "bempp-cl_b200", "csrc")
SOURCES = {name: open(os.path.join(CSRC, name)).read() for name in sorted(os.listdir(CSRC))
           if name.endswith((".cu", ".cuh"))}
CALL = re.compile(r"= park_orbit_trial<[^;]*;")


@pytest.mark.parametrize("name", [n for n, text in SOURCES.items() if CALL.search(text)])
def test_parked_fields_are_fenced(name):
    """The loads of a parked trial element name no memory: a fence stands between the last store and the first load."""
    text = SOURCES[name]
    for call in CALL.finditer(text):
        rest = text[call.end():]
        fence = rest.find("orbit_fence();")
        assert fence >= 0
        assert not re.search(r"\.(ld|li|f|n)\(|orbit_pair<|pair_sym64<", rest[:fence])
        stores = [m.start() for m in re.finditer(r"park\[[^\n]*\] = ", rest)]
        assert all(at < fence for at in stores)


def test_only_the_parked_fields_are_read_without_naming_memory():
    for name, text in SOURCES.items():
        for statement in re.findall(r"asm[^;]*?\((.*?)\);", text, re.S):
            if re.search(r"\b(ld|st)\.(volatile\.)?shared", statement):
                assert '"memory"' in statement or name == "orbit_pair.cuh", statement

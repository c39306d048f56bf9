"""A kernel that gives up on a bounded wait leaves a number in the device's error word: it has to name one place."""
import collections
import os
import re

from conftest import CSRC


def test_every_error_code_belongs_to_one_file():
    places = collections.defaultdict(set)
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh", ".h")):
            with open(os.path.join(CSRC, name)) as f:
                for code in re.findall(r"atomicExch\(\s*(?:p\.)?err\s*,\s*(\d+)\s*\)|p\.err\s*,\s*(\d+)\s*\)", f.read()):
                    places[int(code[0] or code[1])].add(name)
    assert len(places) > 20
    shared = {code: sorted(names) for code, names in places.items() if len(names) > 1}
    assert not shared, shared

"""A scan whose look-back outwaits its bound leaves sums that are too small, a sort
places that were not written, and both are places in memory. (Read from the source:
no input makes a wait run out.) Host code checks the error word with every read
back of sizes, and of the kernels that work on the device's own the first after each
scan or sort looks at it."""

import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "galactic-tides_gb300" / "csrc"


def body(path, name):
    text = re.sub(r"//[^\n]*", "", (CSRC / path).read_text())
    start = text.index("{", re.search(rf"\b{name}\s*(=\s*\[&\])?\(", text).end())
    depth, end = 1, start + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
    return text[start:end]


@pytest.mark.parametrize("path,name,check", [
    ("tree_build.cu", "read_scalars", "check_device_error(host->error)"),
    ("group_walk.cu", "read_scalars", "check_device_error(host->error)"),
    ("learned_walk.cu", "read_back", "check_device_error(flags[1])"),
    ("tree_build.cu", "k_check_tree_graph", "sc->error"),     # the node count's scan
    ("group_walk.cu", "k_check_groups_graph", "sc->error"),   # the groups'
    ("learned_walk.cu", "k_lrows", "sc->error"),              # the deferred pairs'
    ("tree_build.cu", "k_levels", "sc->error"),               # the keys' sort
    ("tree_build.cu", "k_forest_sys_keys", "*error"),         # a forest's, by key
    ("tree_build.cu", "k_forest_gather", "*error"),           # and by system
    ("tree_build.cu", "k_seg_keys", "*error"),                # the deeper keys', by word
    ("tree_build.cu", "k_deep_scatter", "*error"),            # and by segment
])
def test_errors_are_seen_before_places_are_used(path, name, check):
    assert check in body(path, name)

"""What a kernel may touch before it waits for the kernel in front of it.

Launched with programmatic stream serialization a kernel may start while the one in front still runs, and only
griddepcontrol.wait makes what that one wrote visible.  Before the wait a kernel reads nothing but packed weights
with their scales and biases, which the caller must have written earlier (include/metile_b200.h).  Checked in the
source: a read that comes too early is a race, which no run has to show."""

import glob
import os
import re

import pytest

from metile_b200 import build

IN_THE_PARAMETERS = {"p.w_map", "p.w", "p.peers"}  # arrays of the parameter block itself


def kernels():
    for path in sorted(glob.glob(os.path.join(build.CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*|__launch_bounds__\([^)]*\)", "", open(path).read())
        for match in re.finditer(r"__global__\s+void[^;{]*?(\w+)\(([^;{]*?)\)\s*\{", text):
            body, depth, at = "", 1, match.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                body += text[at]
                at += 1
            if "griddep_wait" in body:
                yield pytest.param(match.group(2), body.split("griddep_wait")[0], id=match.group(1))


@pytest.mark.parametrize("parameters,before", list(kernels()))
def test_only_weights_are_read_before_the_wait(parameters, before):
    pointers = set(re.findall(r"\*\s*(?:__restrict__\s*)?(\w+)", parameters))
    touched = {name for name in re.findall(r"(\bp\.\w+|\b\w+)\s*\[", before) if name in pointers or name.startswith("p.")}
    touched |= set(re.findall(r"(?:ld_global_\w+|__ldg|cp_async_\d+)\([^;]*?(\bp\.\w+)", before))
    assert touched <= IN_THE_PARAMETERS


def test_the_kernels_were_found():
    assert len(list(kernels())) >= 10

"""A kernel that gave up a wait may not end with bulk copies in flight: they would land
in shared memory that another block holds by then.  No wait can be made to expire in
these kernels without a fault, so this is held to in the source: behind its last
asynchronous load each has the (bounded) wait for what has not landed."""
import os
import re

import pytest

from conftest import ROOT


def kernel(file, name):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(ROOT, "marl-ochre_b200", "csrc", file)).read())
    at = text.index("{", text.index(name + "("))
    depth, end = 1, at + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
    return text[at:end]


@pytest.mark.parametrize("file,name,load,drain", [
    ("mlp_train.cu", "k_train_rows", "image_load(", "image_loads_drain("),
    ("mlp_train.cu", "k_train_weights", "load(next)", "image_loads_drain("),
    ("field.cu", "void diffuse_tile", "issue(", "mbar_wait_bounded(&bars[q % STAGES]"),
])
def test_drained(file, name, load, drain):
    body = kernel(file, name)
    assert drain in body[body.rindex(load):], name

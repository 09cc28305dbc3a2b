"""Dependent launches (common.cuh): a kernel reads nothing that an earlier launch
wrote before griddep_wait(), or says that it does by reads_before_wait().

What a read too early would give depends on what else runs, so the rule is held to
in the source: in the body of every kernel that waits, what stands before the first
wait may use no pointer argument unless reads_before_wait() stands before it.
"""
import glob
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "marl-ochre_b200", "csrc")

# Reads ahead of the wait that no launch in flight can have written.
ALLOWED = {"k_train_rows": {"a"}}  # the batch's row indices (launch arguments) and X, which is written before training


def kernels():
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void[^{;]*?\b(k_\w+)\s*\(([^{;]*)\)\s*\{", text):
            depth, end = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            found.append((m.group(1), m.group(2), text[m.end():end]))
    return found


WAITING = [k for k in kernels() if "griddep_wait()" in k[2]]


def test_all_waiting_kernels_are_found():
    names = {k[0] for k in WAITING}
    assert {"k_fate_scatter", "k_fate_resolve", "k_fate_moves", "k_fate_births", "k_train_rows", "k_train_weights",
            "k_train_update", "k_diffuse_batch", "k_light", "k_light_batch"} <= names


@pytest.mark.parametrize("name,params,body", WAITING, ids=[k[0] for k in WAITING])
def test_reads_before_the_wait(name, params, body):
    before = body[:body.index("griddep_wait()")]
    before = before.split("reads_before_wait()")[0]
    args = {re.search(r"(\w+)\s*$", p).group(1) for p in params.split(",")} - ALLOWED.get(name, set())
    used = {a for a in args if re.search(r"\b%s\s*(\.|->|\[)" % a, before)}
    assert not used, (name, used)


def test_the_kernel_before_an_early_reader_waits_before_it_triggers():
    bodies = {k[0]: k[2] for k in kernels()}
    for reader, before in (("k_fate_births", "k_fate_moves"), ("k_train_update", "k_train_weights"),
                           ("k_train_update", "k_train_rows")):
        if "reads_before_wait()" in bodies[reader]:
            body = bodies[before]
            assert body.index("griddep_wait()") < body.index("griddep_launch_dependents()"), before

"""The four-lane cell loop's hand-over between lanes, held to in the source.

A group's lanes acquire different dependencies and the group's other lanes read what
those cells scattered; a publishing lane releases what the others stored.  Votes order
no memory, so a __syncwarp() has to stand between in either direction.  What a missing
one gives depends on the compiler and the chip, and no run shows it.
"""
import os
import re

from conftest import ROOT

TEXT = re.sub(r"//[^\n]*", "", open(os.path.join(ROOT, "marl-ochre_b200", "csrc", "cells_quad.cuh")).read())


def body(name):
    at = TEXT.index("{", TEXT.index(name + "("))
    depth, end = 1, at + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(TEXT[end], 0)
        end += 1
    return TEXT[at:end]


def test_acquires_reach_the_lanes_that_gather():
    loop = body("void quad_loop")
    assert "__syncwarp();" in loop[loop.rindex("ld_acquire_u32("):loop.index("quad_update(")]


def test_stores_reach_the_lane_that_publishes():
    update = body("bool quad_update")
    assert "__syncwarp();" in update[update.rindex("st4("):update.index("st_release_u32(")]

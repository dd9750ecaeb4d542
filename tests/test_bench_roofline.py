"""The bench's roofline block: a phase's bytes and traffic cover every kernel
that its time covers."""
import json
import os

import pytest

import bench


@pytest.mark.parametrize("phase,kernels", [("union", ("k_link", "k_union")), ("decrement", ("k_decr",)),
                                           ("increment", ("k_incr",)), ("label", ("k_border",)), ("merge", ("k_merge",))])
def test_traffic_covers_the_phases_kernels(phase, kernels):
    with open(os.path.join(bench.ROOT, "profiles", "ncu_traffic.json")) as f:
        per_kernel = json.load(f)
    assert bench.ncu_traffic(phase) == sum(per_kernel[k] for k in kernels)


def test_union_bytes_are_the_link_and_the_union_pass():
    assert bench.algorithmic_bytes("union", 1_000, 10, 3, 0, 0) == 2 * 28 * 1_000
    avg = {"merge": 0.02, "union": 0.15}
    st = {"chunks_per_slide": 1, "cells": 0, "work_items": 0}
    block = bench.roofline_block(avg, st, {"cluster_tests": 0, "query_tests": 0}, 1_000, 10, 0.3, 6_777.0, "measured")
    assert block["kernels"] == ["k_link", "k_union"]
    assert block["algorithmic_bytes_per_launch"] == 56_000

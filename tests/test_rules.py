"""The host rules of kds_rules.h, without a device."""
import itertools
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    out = str(tmp_path_factory.mktemp("rules") / "rules_main")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Wextra", "-Werror", "-I",
                    os.path.join(ROOT, "kd_slam2_b200", "csrc"), os.path.join(ROOT, "tests", "cpp", "rules_main.cpp"),
                    "-o", out], check=True, capture_output=True, text=True)

    def call(*args):
        r = subprocess.run([out, *map(str, args)], check=True, capture_output=True, text=True)
        return [int(x) for x in r.stdout.split()]
    return call


def test_first_stamp_kernel_runs_on_the_servers_device_only(rules):
    """The kernel's scratch is on the server's device: a caller whose current device and arrays
    are on another one takes the copy (the kernel would write memory that it cannot reach)."""
    for current, server, first, last in itertools.product((0, 1), repeat=4):
        same = current == server == first == last
        assert rules("first_stamp", current, server, first, last) == [1 if same else 0]


@pytest.mark.parametrize("room,blocks", [(0, 0), (7, 0), (8, 8), (15, 8), (16, 16), (64, 16)])
def test_alignments_need_no_cluster(rules, room, blocks):
    """Where the device schedules no cluster the rule says so (and an alignment is launched once
    per iteration) instead of assuming that the portable size always fits."""
    assert rules("cluster", room) == [blocks]


def test_kernel_limits_are_set_on_every_device(rules):
    """A limit raised on one device says nothing of the next one."""
    assert rules("devices", 0, 0, 1, 0, 1, 63, 63, 64, 64, -1, -1) == [1, 0, 1, 0, 0, 1, 0, 1, 1, 1, 1]

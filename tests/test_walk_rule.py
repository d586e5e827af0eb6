"""When a walk's groups get two warps each: the rule compiled for the host.  A
caller's occupancy (walk_blocks_per_sm) always means the one-warp kernel; small
batches and leaves do too, and for many groups a wide opening angle."""
import os
import subprocess

import pytest

from conftest import PKG, ROOT

SOURCE = """
#include <cstdio>
#include "gcs_internal.h"
int main() {
    int groups, sms, bps, batch, leaf;
    float theta;
    while (scanf("%d %d %d %d %d %f", &groups, &sms, &bps, &batch, &leaf, &theta) == 6)
        printf("%d\\n", gcs::walk_pairs_pay(groups, sms, bps, batch, leaf, theta * theta) ? 1 : 0);
}
"""

CASES = [  # groups, SMs, blocks per SM -> two warps
    (1, 148, 0, 1), (44, 148, 0, 1), (1408, 148, 0, 1), (100000, 148, 0, 0),
    (1, 148, 1, 0), (44, 148, 4, 0), (1408, 148, 8, 0), (100000, 148, 2, 0),
]


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("rule")
    (d / "rule.cpp").write_text(SOURCE)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(PKG, "csrc"), "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(cuda, "include"), "-o", str(d / "rule"), str(d / "rule.cpp")], check=True)

    def ask(*numbers):
        out = subprocess.run([str(d / "rule")], input=" ".join(map(str, numbers)), capture_output=True, text=True,
                             check=True).stdout
        return int(out)
    return ask


@pytest.mark.parametrize("groups,sms,bps,two", CASES)
def test_occupancy_means_one_warp(rule, groups, sms, bps, two):
    assert rule(groups, sms, bps, 64, 8, 0.5) == two


# batch, leaf size, theta, groups an SM up to which two warps walk a group
LINES = [(64, 8, 0.5, 20), (64, 4, 0.5, 15), (64, 1, 0.0, 16), (64, 8, 0.75, 13.75), (64, 16, 0.7, 20), (64, 1, 1.0, 12),
         (64, 32, 1.0, 20), (33, 1, 1.0, 12), (32, 8, 0.5, 12), (32, 16, 0.5, 20), (32, 4, 0.7, 6), (32, 1, 1.0, 0),
         (16, 8, 0.5, 6), (16, 16, 1.0, 12), (16, 4, 0.5, 0), (8, 32, 0.5, 12), (8, 8, 0.5, 0), (1, 32, 0.5, 0)]


@pytest.mark.parametrize("batch,leaf,theta,per_sm", LINES)
def test_line(rule, batch, leaf, theta, per_sm):
    for sms in (148, 100):
        assert rule(int(per_sm * sms), sms, 0, batch, leaf, theta) == (1 if per_sm else 0)
        assert rule(int(per_sm * sms) + 1, sms, 0, batch, leaf, theta) == 0

"""Which team solves a single body (csrc/solve_rule.h), for every size of the widest resident cluster."""
import subprocess

import pytest
from conftest import ROOT

from bounce_softbody_gb300 import build

PROGRAM = r"""
#include "solve_rule.h"
#include <cstdio>
#include <initializer_list>
int main()
{
	for (int widest : {0, 1, 2, 4, 8, 16})
		for (int n = 1; n <= 300; ++n) std::printf("%d %d %d\n", widest, n, b3g::cluster_ctas(n, widest));
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("rule")
    (d / "rule.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", build.CSRC, str(d / "rule.cpp"), "-o", str(d / "rule")], check=True)
    out = subprocess.run([str(d / "rule")], check=True, capture_output=True, text=True).stdout
    return [tuple(map(int, line.split())) for line in out.splitlines()]


def test_a_cluster_is_one_the_device_can_hold(rule):
    for widest, n, cl in rule:
        assert cl in (0, 1, 2, 4, 8, 16) and cl <= widest
        assert cl == 0 or n <= 8 * cl <= 8 * widest  # at most eight slices a CTA
        assert cl > 0 or n > 8 * widest              # a body that fits takes one


def test_wide_clusters_take_two_slices_a_cta(rule):
    for widest, n, cl in rule:
        if widest == 16 and n <= 128:
            assert cl == next(c for c in (1, 2, 4, 8, 16) if n <= 2 * c or c == 16)

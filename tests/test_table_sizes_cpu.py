"""Sizes of hash tables (csrc/qm_slots.h), compiled for the host: a stream's
table grows to a power of two for its groups, and a stream of more groups than
a table may have slots for is refused ahead of any work."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "querymode_b200", "csrc")

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "qm_slots.h"
int main(int argc, char **argv) {
  for (int i = 1; i + 1 < argc; i += 2)
    std::printf("%lld %d\n", (long long)qm_hash_slots(atoll(argv[i])), qm_grown_log2(atoll(argv[i]), atoll(argv[i + 1])));
}
"""


@pytest.fixture(scope="module")
def sizes(tmp_path_factory):
    d = tmp_path_factory.mktemp("slots")
    (d / "slots.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(d / "slots.cpp"), "-o", str(d / "slots")], check=True)

    def get(groups, n_slots):
        out = subprocess.run([str(d / "slots"), str(groups), str(n_slots)], check=True, capture_output=True, text=True).stdout.split()
        return int(out[0]), int(out[1])
    return get


@pytest.mark.parametrize("groups,n_slots,one_shot,grown", [
    (1, 1024, 1024, 0), (482, 1024, 1024, 0), (483, 1024, 1026, 11), (20_000, 1024, 42_500, 16), (20_000, 65_536, 42_500, 0),
    (1_010_580_540, 1 << 31, 2_147_483_647, 0), (1_010_580_541, 1 << 31, 1 << 31, 32), (1 << 32, 1 << 31, 1 << 31, 34),
    (1 << 40, 1024, 1 << 31, 42)])
def test_sizes(sizes, groups, n_slots, one_shot, grown):
    assert sizes(groups, n_slots) == (one_shot, grown)


def test_growth_is_refused_past_the_largest_table():
    with open(os.path.join(CSRC, "qm_api.cu")) as f:
        api = f.read()
    grow = api[api.index("int grow_table("):]
    assert grow.index("log2cap > QM_MAX_LOG2_SLOTS) return set_err") < grow.index("ensure(")

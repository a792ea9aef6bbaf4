"""Index rules of the kernels and launchers (csrc/share_rules.hpp), compiled for the host with the warnings that catch an order of
evaluation left to the compiler."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "apathy-atlas_b200", "csrc")

SOURCE = """
#include "share_rules.hpp"
extern "C" uint32_t next_own_granule(uint32_t g, uint32_t ks) { return atlas::next_own_granule(g, ks); }
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "rules.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", "-shared", "-fPIC", f"-I{CSRC}", "-o", str(d / "rules.so"), str(d / "rules.cpp")],
                   check=True)
    return C.CDLL(str(d / "rules.so"))


@pytest.mark.parametrize("ks", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("n_gran", [0, 1, 3, 4, 5, 8, 31, 64, 127, 2048])
def test_granules_of_a_k_split(rules, ks, n_gran):
    """Every granule is one CTA's, in blocks of four, each CTA's ascending."""
    taken = {}
    for kz in range(ks):
        g = 4 * kz
        before = -1
        while g < n_gran:
            assert g > before and g not in taken
            taken[g] = kz
            before, g = g, rules.next_own_granule(g, ks)
    assert taken == {g: (g // 4) % ks for g in range(n_gran)}

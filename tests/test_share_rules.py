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
extern "C" void mma_shrink_grid(uint32_t slots, uint32_t granules, uint32_t chunks, uint32_t rows, uint32_t sms, int beside, uint32_t* out) {
    const atlas::MmaShrinkGrid g = atlas::mma_shrink_grid(slots, granules, chunks, rows, sms, atlas::MachineBeside(beside));
    out[0] = g.ksplit; out[1] = g.row_parts_log2; out[2] = g.prefetch_ctas;
}
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


NONE, PART, ALL = 0, 1, 2       # of the machine wanted by a dependent beside the grid


def _grid(rules, slots, granules, chunks, rows, beside, sms=148):
    out = (C.c_uint32 * 3)()
    rules.mma_shrink_grid(slots, granules, chunks, rows, sms, beside, out)
    return tuple(out)


@pytest.mark.parametrize("slots,granules,chunks", [(1, 1, 1), (1, 8, 4), (2, 1, 4), (8, 1, 2), (8, 4, 2), (16, 1, 4), (37, 2, 1), (64, 4, 1), (4096, 8, 4)])
@pytest.mark.parametrize("rows", [1, 32, 33, 130, 256])
@pytest.mark.parametrize("beside", [NONE, PART, ALL])
def test_grid_of_the_mma_shrink(rules, slots, granules, chunks, rows, beside):
    """Row parts stay within what can be resident, and beside a kernel that wants the machine within half of it where more would mostly
    be CTAs without rows."""
    items, resident = slots * granules * chunks, 148 * 8
    ksplit, log2, first = _grid(rules, slots, granules, chunks, rows, beside)
    assert first == resident and ksplit in ((2, 4, 8) if beside == PART else (8,))
    if ksplit < 8:
        assert items * 2 * ksplit > resident // 2
    if log2:
        ctas = items * ksplit << log2
        assert 32 << (log2 - 1) < rows and ctas <= resident
        assert ctas <= resident // 2 or beside != ALL or rows >= slots * 32 << (log2 - 1) or chunks == 1 or (log2 == 1 and chunks == 2)


def test_clusters_without_rows_do_not_fill_the_machine(rules):
    assert _grid(rules, 8, 1, 2, 256, ALL)[:2] == (8, 2)       # 512 tokens of 8 adapters of rank 16: 512 CTAs, not 1024
    assert _grid(rules, 8, 1, 4, 256, ALL)[:2] == (8, 1)       # 1000 tokens of them
    assert _grid(rules, 16, 1, 4, 256, ALL)[:2] == (8, 0)      # ... of 16
    assert _grid(rules, 8, 4, 2, 256, ALL)[:2] == (8, 1)       # rank 64, two chunks: two clusters
    assert _grid(rules, 1, 8, 4, 256, ALL)[:2] == (8, 2)       # one adapter for all rows: 1024 CTAs with rows
    assert _grid(rules, 8, 1, 4, 256, NONE)[:2] == (8, 2)


@pytest.mark.parametrize("slots,granules,chunks", [(1, 1, 1), (1, 8, 4), (8, 4, 2), (8, 4, 4), (8, 8, 2), (16, 1, 4), (64, 4, 1), (128, 1, 1), (4096, 8, 4)])
@pytest.mark.parametrize("rows", [1, 32, 33, 130, 256])
def test_one_more_cluster_beside_a_kernel_of_one_tile_a_cta(rules, slots, granules, chunks, rows):
    TILES = 3
    ksplit, log2, first = _grid(rules, slots, granules, chunks, rows, TILES)
    assert (ksplit, first) == (8, 148 * 8)
    if log2 != _grid(rules, slots, granules, chunks, rows, ALL)[1]:
        assert log2 == 1 and rows > 32 and slots * granules * chunks * 16 <= 2 * 148 * 8
        assert chunks <= 2 or rows >= slots * 32
    if (slots, granules, chunks, rows) == (8, 4, 4, 256):      # 1000 tokens of 8 adapters of rank 64
        assert log2 == 1

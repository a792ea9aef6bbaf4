"""Operands handed over in groups: four K blocks of the expanded weights, two of the activations, blocks of two or four LoRA granules with one,
two or four of B_s in a copy.  Lengths that leave part of a group, rings that wrap and lists whose slots straddle a block, on scratch
that holds garbage: within the path's tolerance of the oracle, and the same bits call for call and form for form."""
import numpy as np
import pytest

from gpu_util import DeviceCase, assert_close, ideal

pytestmark = pytest.mark.gpu

MIXED = [16, 64, 8, 48, 32, 64, 16, 24, 56, 64, 40, 16]


def _sample(case, seed):
    rng = np.random.default_rng(seed)
    pick = lambda n, k: np.sort(rng.choice(n, min(n, k), replace=False)).astype(np.uint32)
    return pick(case.M, 48), pick(case.N, 96)


# K blocks of 64: 4, 8, 12, 20, 36 of them, and 5, 7, 8 (the last half full), 12 (half full), 45
@pytest.mark.parametrize("form", ["", "single", "unsplit"])
@pytest.mark.parametrize("K", [256, 512, 768, 1280, 2304, 288, 416, 480, 736, 2880])
@pytest.mark.parametrize("M", [20, 60, 130, 250])
def test_every_length_of_the_base_loop(cuda, atlas, oracle, M, K, form):
    from atlas_b200 import synth
    case = synth.make_case("groups", M=M, K=K, N=376, ranks=MIXED, max_rank=64, max_loras=13, none_frac=0.15, scale2=0.02, b_std=0.1, seed=M + K)
    dc = DeviceCase(cuda, atlas, case)
    flags = {"": 0, "single": atlas.FLAG_NO_CTA_PAIR, "unsplit": atlas.FLAG_NO_K_SPLIT}[form]
    y, variant = dc.run(flags=flags, lora_ws=True)
    assert variant == atlas.VARIANT_TCGEN05
    rows, cols = _sample(case, K)
    assert_close(oracle, y[np.ix_(rows, cols)], ideal(oracle, case, rows=rows, cols=cols), form)
    for _ in range(3):                                   # fresh scratch every time
        assert np.array_equal(dc.run(flags=flags, lora_ws=True)[0], y)
    assert atlas.device_status() == 0


# 256-token tiles by single CTAs: a ring of four stages of one K block, beside groups of four, that wraps before the expansion has waited for it
@pytest.mark.parametrize("K", [1280, 2560, 4096])
def test_a_ring_of_single_blocks(cuda, atlas, oracle, K):
    from atlas_b200 import synth
    case = synth.make_case("single_blocks", M=256, K=K, N=8704, ranks=[32] * 16, max_rank=32, none_frac=0.1, scale2=0.02, b_std=0.1, seed=K)
    dc = DeviceCase(cuda, atlas, case)
    y, _ = dc.run(flags=atlas.FLAG_NO_CTA_PAIR, lora_ws=True)
    assert not atlas.last_launch_shape()["cta_pair"]
    rows, cols = _sample(case, K)
    assert_close(oracle, y[np.ix_(rows, cols)], ideal(oracle, case, rows=rows, cols=cols), "single")
    for _ in range(5):
        assert np.array_equal(dc.run(flags=atlas.FLAG_NO_CTA_PAIR, lora_ws=True)[0], y)
    assert atlas.device_status() == 0


@pytest.mark.parametrize("fp4", [False, True])
@pytest.mark.parametrize("ranks,max_rank,ids", [
    ([16] * 45, 16, "uniform"),                          # one granule a slot, the last block part full
    ([32, 16, 32, 32, 16] * 7, 32, "uniform"),           # copies of two, some slots off their boundary
    (MIXED * 3, 64, "uniform"),                          # copies of four (two in one-tile BF16 passes)
    ([64] * 3, 64, "segments"),
])
def test_lora_blocks_of_the_persistent_kernel(cuda, atlas, oracle, ranks, max_rank, ids, fp4):
    from atlas_b200 import synth
    case = synth.make_case("blocks", M=2085, K=512, N=4864, ranks=ranks, max_rank=max_rank, max_loras=len(ranks) + 2, ids=ids, segments=24,
                           none_frac=0.15, scale2=0.02, b_std=0.1, seed=len(ranks) + max_rank)
    dc = DeviceCase(cuda, atlas, case)
    mode = atlas.FLAG_ACT_FP4 if fp4 else 0
    y, _ = dc.run(flags=mode, lora_ws=True)
    assert atlas.last_launch_shape()["persistent_tiles_per_pass"] == (1 if fp4 else 2)
    one, _ = dc.run(flags=mode | atlas.FLAG_ONE_TILE_PASS, lora_ws=True)
    assert atlas.last_launch_shape()["persistent_tiles_per_pass"] == 1
    tile, _ = dc.run(flags=mode | atlas.FLAG_NO_PERSISTENT, lora_ws=True)
    assert np.array_equal(y, one) and np.array_equal(y, tile)
    rows, cols = _sample(case, max_rank)
    assert_close(oracle, y[np.ix_(rows, cols)], ideal(oracle, case, rows=rows, cols=cols, act_fp4=fp4), "blocks")
    assert atlas.device_status() == 0


# two and three CTAs to a tile's K beside the shrink, pairs (with gaps) and single CTAs: rings that wrap with the stage before waited for
@pytest.mark.parametrize("form", ["", "single"])
@pytest.mark.parametrize("M,K,N", [(400, 4608, 4096), (512, 6400, 2560), (300, 4352, 4090)])
def test_gaps_for_the_shrink(cuda, atlas, oracle, M, K, N, form):
    from atlas_b200 import synth
    case = synth.make_case("gaps", M=M, K=K, N=N, ranks=[32, 16, 8, 24], max_rank=32, none_frac=0.15, scale2=0.02, b_std=0.1, seed=M + K)
    dc = DeviceCase(cuda, atlas, case)
    flags = atlas.FLAG_NO_CTA_PAIR if form else 0
    y, _ = dc.run(flags=flags, lora_ws=True)
    shape = atlas.last_launch_shape()
    assert shape["token_tile"] == 256 and shape["k_split"] in (2, 3), shape
    assert shape["gaps_for_shrink"] == shape["cta_pair"] and shape["cta_pair"] == (form == ""), shape
    rows, cols = _sample(case, K)
    assert_close(oracle, y[np.ix_(rows, cols)], ideal(oracle, case, rows=rows, cols=cols), form)
    for _ in range(3):
        assert np.array_equal(dc.run(flags=flags, lora_ws=True)[0], y)
    assert atlas.device_status() == 0


# either side of the lines: K, CTAs to a tile's K, granules, tokens, pairs, a shrink to run beside
@pytest.mark.parametrize("M,K,N,ads,max_rank,flags,gaps", [
    (1000, 4352, 4096, 4, 32, 0, True), (1000, 4096, 4096, 4, 32, 0, False), (1000, 4352, 4096, 1, 16, 0, False),
    (1000, 4352, 4096, 17, 32, 0, False), (256, 4352, 14336, 4, 32, 0, False), (260, 4352, 8192, 4, 32, 0, True), (512, 4352, 2560, 4, 32, 0, False), (512, 6400, 1024, 4, 32, 0, False),
    (400, 4608, 4096, 16, 64, 0, True), (400, 4608, 4096, 65, 16, 0, False), (400, 4608, 4096, 1, 8, 0, True), (300, 4608, 4096, 2, 16, "single", False),
    (400, 4608, 4096, 2, 16, "base", False), (1030, 4352, 1000, 2, 16, 0, False)])
def test_which_calls_leave_gaps(cuda, atlas, oracle, M, K, N, ads, max_rank, flags, gaps):
    from atlas_b200 import synth
    case = synth.make_case("gap_lines", M=M, K=K, N=N, ranks=[max_rank] * ads, max_rank=max_rank, none_frac=0.15, scale2=0.02, b_std=0.1, seed=M + ads)
    dc = DeviceCase(cuda, atlas, case)
    y, _ = dc.run(flags=atlas.FLAG_NO_CTA_PAIR if flags == "single" else 0, lora_ws=True, lora=flags != "base")
    assert atlas.last_launch_shape()["gaps_for_shrink"] == gaps, atlas.last_launch_shape()
    rows, cols = _sample(case, K)
    assert_close(oracle, y[np.ix_(rows, cols)], ideal(oracle, case, rows=rows, cols=cols, lora=flags != "base"), "gaps")
    assert atlas.device_status() == 0

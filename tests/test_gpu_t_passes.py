"""The persistent form: wide fetches of B_s, block scales of two K blocks at a time; granule lists and shrink splits at their edges.

Tolerances: the path's own against the FP32-accumulated oracle (gpu_util); bits where two forms add in the same order."""
import numpy as np
import pytest

from gpu_util import DeviceCase, assert_close, ideal

pytestmark = pytest.mark.gpu


def _sample(case, n_rows, n_cols, seed):
    rng = np.random.default_rng(seed)
    rows = np.sort(rng.choice(case.M, min(case.M, n_rows), replace=False)).astype(np.uint32)
    cols = np.sort(rng.choice(case.N, min(case.N, n_cols), replace=False)).astype(np.uint32)
    return rows, cols


@pytest.mark.parametrize("fp4", [False, True])
@pytest.mark.parametrize("max_rank,ranks", [
    (16, [16, 8, 16]), (32, [32, 16, 8]), (48, [48, 16, 33]), (64, [64, 8, 33, 48]),
])
def test_granules_of_b_fetched_together(cuda, atlas, oracle, max_rank, ranks, fp4):
    """One, two and four granules of a slot per copy, slots that fill it in part, one and two token tiles per pass."""
    from atlas_b200 import synth
    case = synth.make_case("wide", M=2085, K=512, N=4992, ranks=ranks, max_rank=max_rank, max_loras=len(ranks) + 1, none_frac=0.1,
                           scale2=0.02, b_std=0.1, seed=max_rank)
    dc = DeviceCase(cuda, atlas, case)
    mode = atlas.FLAG_ACT_FP4 if fp4 else 0
    one, _ = dc.run(flags=mode | atlas.FLAG_NO_PERSISTENT, lora_ws=True)
    for flags in (mode, mode | atlas.FLAG_ONE_TILE_PASS):
        y, _ = dc.run(flags=flags, lora_ws=True)
        assert atlas.last_launch_shape()["persistent_tiles_per_pass"] > 0
        assert np.array_equal(y, one)
    rows, cols = _sample(case, 48, 64, max_rank)
    assert_close(oracle, one[np.ix_(rows, cols)], ideal(oracle, case, rows=rows, cols=cols, act_fp4=fp4), "sample")
    assert atlas.device_status() == 0


@pytest.mark.parametrize("max_rank,ranks", [(96, [96, 80, 8, 33]), (128, [128, 80, 64, 8])])
def test_granules_of_b_above_rank_64(cuda, atlas, oracle, max_rank, ranks):
    """Several copies to a slot: of two granules (96; one token tile per pass), of four (128, two token tiles).  (FP4 activations take
    ranks up to 64.)"""
    from atlas_b200 import synth
    case = synth.make_case("wide128", M=2085, K=512, N=4992, ranks=ranks, max_rank=max_rank, max_loras=len(ranks) + 1, none_frac=0.1, scale2=0.02,
                           b_std=0.1, seed=4)
    dc = DeviceCase(cuda, atlas, case)
    one, _ = dc.run(flags=atlas.FLAG_NO_PERSISTENT, lora_ws=True)
    assert atlas.last_launch_shape()["persistent_tiles_per_pass"] == 0
    for flags, tiles in ((0, 2), (atlas.FLAG_ONE_TILE_PASS, 1)):
        y, _ = dc.run(flags=flags, lora_ws=True)
        assert atlas.last_launch_shape()["persistent_tiles_per_pass"] == tiles
        assert np.array_equal(y, one)
    rows, cols = _sample(case, 48, 64, 5)
    assert_close(oracle, one[np.ix_(rows, cols)], ideal(oracle, case, rows=rows, cols=cols), "sample")
    assert atlas.device_status() == 0


@pytest.mark.parametrize("K", [256, 512, 768, 1280, 2048])
def test_fp4_scales_of_two_blocks(cuda, atlas, oracle, K):
    """One K block, whole and odd numbers of pairs of them."""
    from atlas_b200 import synth
    case = synth.make_case("scales", M=1030, K=K, N=4992, ranks=[16, 8], max_rank=16, scale2=0.02, b_std=0.1, seed=K)
    dc = DeviceCase(cuda, atlas, case)
    y, _ = dc.run(flags=atlas.FLAG_ACT_FP4, lora_ws=True)
    assert atlas.last_launch_shape()["persistent_tiles_per_pass"] == 1
    one, _ = dc.run(flags=atlas.FLAG_ACT_FP4 | atlas.FLAG_NO_PERSISTENT, lora_ws=True)
    assert np.array_equal(y, one)
    rows, cols = _sample(case, 48, 64, K)
    assert_close(oracle, y[np.ix_(rows, cols)], ideal(oracle, case, rows=rows, cols=cols, act_fp4=True), "sample")
    assert atlas.device_status() == 0


@pytest.mark.parametrize("M,max_loras,stride", [(16, 40, 3), (17, 40, 1), (64, 200, 3), (128, 128, 1), (129, 500, 37), (256, 256, 1)])
def test_granule_list_of_scattered_slots(cuda, atlas, oracle, M, max_loras, stride):
    """Every token its own slot, slots scattered over the bitmap's words, some without an adapter, ranks of one to four granules."""
    from atlas_b200 import synth
    case = synth.make_case("list", M=M, K=512, N=384, ranks=[8], max_rank=64, max_loras=max_loras, scale2=0.02, b_std=0.1, seed=M)
    for s in range(max_loras):
        case.adapters[s] = None if s % 7 == 3 else synth.make_adapter(900 + s % 4, 512, 384, (8, 16, 40, 64)[s % 4], 80.0, 0.02)
    case.seq_slot = ((np.arange(M) * stride + 5) % max_loras).astype(np.int32)
    dc = DeviceCase(cuda, atlas, case)
    y, _ = dc.run(flags=atlas.FLAG_FORCE_TCGEN05, lora_ws=True)
    build, _ = dc.run(flags=atlas.FLAG_FORCE_TCGEN05)
    assert np.array_equal(y, build)
    rows, cols = _sample(case, 64, 96, M)
    assert_close(oracle, y[np.ix_(rows, cols)], ideal(oracle, case, rows=rows, cols=cols), "sample")
    assert atlas.device_status() == 0


@pytest.mark.parametrize("M,K,ads,ids", [
    (1027, 1024, 8, "segments"),           # eight CTAs to 128 rows, two K blocks each
    (1100, 1280, 30, "uniform"),           # ... shares of two and three blocks, more adapters than a pass of theirs holds
    (2100, 1024, 8, "segments"),           # four
    (2100, 512, 40, "uniform"),
    (4400, 512, 8, "segments"),            # two
])
def test_prefill_shrink_splits(cuda, atlas, oracle, M, K, ads, ids):
    """128 rows in a row without an adapter among them; the same bits from every call."""
    from atlas_b200 import synth
    case = synth.make_case("shrink", M=M, K=K, N=256, ranks=[(16, 64, 48, 8)[i % 4] for i in range(ads)], max_rank=64, max_loras=ads + 1, ids=ids,
                           segments=12, none_frac=0.1, scale2=0.02, b_std=0.1, seed=M + K)
    case.seq_slot[256:512] = -1
    dc = DeviceCase(cuda, atlas, case)
    y, _ = dc.run(lora_ws=True)
    assert atlas.last_launch_shape()["lora_tiles_from_shrink"]
    again, _ = dc.run(lora_ws=True)
    assert np.array_equal(y, again)
    rows, cols = _sample(case, 300, 64, M)
    assert_close(oracle, y[np.ix_(rows, cols)], ideal(oracle, case, rows=rows, cols=cols), "sample")
    assert atlas.device_status() == 0


@pytest.mark.parametrize("M,K,N", [(1, 512, 128), (3, 1024, 4096), (16, 4096, 4104), (40, 576, 8192), (100, 512, 2560), (17, 200, 19072), (300, 512, 1000)])
def test_dense_base_beside_its_shrink(cuda, atlas, oracle, M, K, N):
    """K split over eight, four, two and one CTAs, tokens that do not divide by them; the same bits as base and adapters one after the other."""
    from atlas_b200 import synth
    case = synth.make_case("dense", M=M, K=K, N=N, ranks=[16, 8, 32], max_rank=32, base="bf16", none_frac=0.2, b_std=0.1, seed=M + N)
    dc = DeviceCase(cuda, atlas, case)
    y, variant = dc.run()
    assert variant == atlas.VARIANT_TCGEN05
    base, _ = dc.run(lora=False)
    out = cuda.from_numpy(base.view(np.int16).copy()).cuda()
    atlas.apply_lora_bgmv(dc.pool.route(True, True), dc.x, out, dc.seq_slot, M, K, N, dc.lora_t)
    cuda.cuda.synchronize()
    assert np.array_equal(y, out.cpu().numpy().view(np.uint16))
    rows, cols = _sample(case, 32, 128, M)
    assert_close(oracle, y[np.ix_(rows, cols)], ideal(oracle, case, rows=rows, cols=cols), "sample")
    assert atlas.device_status() == 0


@pytest.mark.parametrize("M,K,N", [(1, 512, 9472), (1, 512, 9488), (8, 288, 9500), (7, 1024, 18960), (16, 256, 28672)])
def test_small_batches_of_four_and_eight_warps(cuda, atlas, oracle, M, K, N):
    """Either side of the line between the two, ragged features, K of a part of a step; a token's bits in a batch and alone."""
    from atlas_b200 import synth
    case = synth.make_case("warps", M=M, K=K, N=N, ranks=[16, 8], max_rank=16, scale2=0.02, b_std=0.1, seed=N)
    dc = DeviceCase(cuda, atlas, case)
    y, _ = dc.run()
    assert atlas.last_launch_shape()["token_tile"] == 8
    rows, cols = _sample(case, 16, 512, N)
    assert_close(oracle, y[np.ix_(rows, cols)], ideal(oracle, case, rows=rows, cols=cols), "sample")
    whole_x, whole_slot = case.x, case.seq_slot
    case.M, case.x, case.seq_slot = 1, whole_x[M - 1:], whole_slot[M - 1:]
    alone, _ = DeviceCase(cuda, atlas, case).run()
    assert np.array_equal(alone[0], y[M - 1])
    assert atlas.device_status() == 0


@pytest.mark.parametrize("M,max_rank", [(1, 16), (7, 64), (8, 64), (13, 32), (16, 16)])
def test_small_batches_have_the_bits_of_any_pool(cuda, atlas, oracle, M, max_rank):
    """Four warps to a CTA (a pool of two slots, no pool at all) and, from seven tokens on, eight (one of twenty): the same partial sums."""
    from atlas_b200 import synth
    case = synth.make_case("pools", M=M, K=4352, N=9488, ranks=[max_rank, 8], max_rank=max_rank, none_frac=0.3, scale2=0.02, b_std=0.1, seed=M)
    if M > 2:
        case.seq_slot[:3] = (0, 1, -1)
    small, _ = DeviceCase(cuda, atlas, case).run()
    assert atlas.last_launch_shape()["token_tile"] == 8
    case.max_loras, case.adapters = 20, list(case.adapters) + [None] * 18
    dc = DeviceCase(cuda, atlas, case)
    large, _ = dc.run()
    assert atlas.last_launch_shape()["token_tile"] == 8
    assert np.array_equal(small, large)
    base, _ = dc.run(lora=False)
    none = case.seq_slot < 0
    assert np.array_equal(large[none], base[none])
    rows, cols = _sample(case, 16, 256, M)
    assert_close(oracle, large[np.ix_(rows, cols)], ideal(oracle, case, rows=rows, cols=cols), "sample")
    assert atlas.device_status() == 0


@pytest.mark.parametrize("M,ads", [(33, 1), (64, 1), (65, 2), (130, 1), (256, 2), (257, 1), (700, 3)])
def test_many_rows_of_a_slot(cuda, atlas, oracle, M, ads):
    """Passes of 32 rows shared by several clusters: whole and partial last passes, masked tiles and rows of t."""
    from atlas_b200 import synth
    case = synth.make_case("rows", M=M, K=512, N=384, ranks=[16, 40, 8][:ads], max_rank=40, max_loras=ads, ids="segments", segments=ads,
                           none_frac=0.05, scale2=0.02, b_std=0.1, seed=M)
    dc = DeviceCase(cuda, atlas, case)
    y, _ = dc.run(flags=atlas.FLAG_FORCE_TCGEN05, lora_ws=True)
    build, _ = dc.run(flags=atlas.FLAG_FORCE_TCGEN05)
    assert np.array_equal(y, build)
    rows, cols = _sample(case, 64, 96, M)
    assert_close(oracle, y[np.ix_(rows, cols)], ideal(oracle, case, rows=rows, cols=cols), "sample")
    assert atlas.device_status() == 0


@pytest.mark.parametrize("M,K,N,no_split", [(1100, 256, 128, False), (1025, 256, 640, False), (1500, 1024, 384, True), (2000, 512, 256, True)])
def test_many_tokens_of_a_short_tile(cuda, atlas, oracle, M, K, N, no_split):
    """More than 1024 tokens where few features leave token tiles of 64: masked tiles of that height, as with rows of t."""
    from atlas_b200 import synth
    case = synth.make_case("short", M=M, K=K, N=N, ranks=[16, 64, 8], max_rank=64, max_loras=4, ids="segments", segments=9, none_frac=0.1,
                           scale2=0.02, b_std=0.1, seed=M)
    dc = DeviceCase(cuda, atlas, case)
    flags = atlas.FLAG_NO_K_SPLIT if no_split else 0
    y, _ = dc.run(flags=flags, lora_ws=True)
    shape = atlas.last_launch_shape()
    assert shape["token_tile"] == 64 and shape["lora_tiles_from_shrink"]
    build, _ = dc.run(flags=flags)
    rows, cols = _sample(case, 200, 64, M)
    want = ideal(oracle, case, rows=rows, cols=cols)
    assert_close(oracle, y[np.ix_(rows, cols)], want, "tiles")
    assert_close(oracle, build[np.ix_(rows, cols)], want, "rows of t")
    assert atlas.device_status() == 0

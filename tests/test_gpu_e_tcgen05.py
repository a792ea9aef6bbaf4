"""The tcgen05 path of the fused layer against the FP32-accumulated oracle."""
import numpy as np
import pytest

from gpu_util import DeviceCase, assert_close, ideal

pytestmark = pytest.mark.gpu


def _tc(atlas):
    return atlas.FLAG_FORCE_TCGEN05


def test_decode_through_the_mma_is_bit_exact(cuda, atlas, oracle):
    """One-hot activations: y[m, f] = w[f, m] exactly, so the in-kernel E2M1 x E4M3 expansion is
    compared bit for bit with the oracle's decode (all 16 codes, normal and subnormal scale bytes)."""
    from atlas_b200 import synth
    K, N = 256, 256
    packed, scales = synth.make_nvfp4_weight(31, N, K)
    scales[:, 0] = np.arange(N, dtype=np.uint8) % 0x7F               # every finite scale byte incl. subnormals
    packed[0, :8] = np.arange(8, dtype=np.uint8) | ((np.arange(8, dtype=np.uint8) + 8) << 4)
    x = np.zeros((K, K), dtype=np.float32)
    x[np.arange(K), np.arange(K)] = 1.0
    case = synth.Case("onehot", K, K, N, 8, 1, oracle.f32_to_bf16(x), np.full(K, -1, np.int32), [None],
                      packed=packed, scales=scales, scale2=1.0)
    y, variant = DeviceCase(cuda, atlas, case).run(lora=False, flags=_tc(atlas))
    assert variant == atlas.VARIANT_TCGEN05
    want = oracle.dequant_nvfp4_to_bf16(packed, scales, 1.0, N, K).T     # [K, N]
    # a sum of signed zeros is +0: a weight of -0.0 legitimately comes out as +0.0
    want = np.where(want == 0x8000, 0, want)
    assert np.array_equal(y, want)
    assert atlas.device_status() == 0


@pytest.mark.parametrize("M,K,N", [(16, 256, 128), (40, 512, 200), (64, 1024, 384), (100, 768, 256),
                                   (256, 512, 128), (300, 256, 264), (1, 256, 128)])
def test_base_linear(cuda, atlas, oracle, M, K, N):
    from atlas_b200 import synth
    case = synth.make_case("base", M=M, K=K, N=N, ranks=[8], max_rank=8, scale2=0.02, seed=M + K)
    dc = DeviceCase(cuda, atlas, case, out_row_stride=N + 8)
    y, variant = dc.run(lora=False, flags=_tc(atlas))
    assert variant == atlas.VARIANT_TCGEN05
    assert_close(oracle, y[:, :N], ideal(oracle, case, lora=False), "base")
    assert (y[:, N:] == 0x7FC0).all()
    assert atlas.device_status() == 0


@pytest.mark.parametrize("M,K,N,ranks,max_rank,with_ranks", [
    (16, 256, 128, [16] * 4, 16, True),
    (64, 512, 256, [8, 16, 32, 64] * 8, 64, True),      # heterogeneous ranks, many adapters per tile
    (64, 512, 256, [8, 16, 32, 64] * 8, 64, False),     # contraction over max_rank (no rank table)
    (300, 512, 384, [32] * 16, 32, True),                # two token tiles, the second one partial
    (130, 256, 200, [8, 24], 24, True),                  # max_rank not a multiple of 16, N not of 128
])
def test_fused_lora(cuda, atlas, oracle, M, K, N, ranks, max_rank, with_ranks):
    from atlas_b200 import synth
    case = synth.make_case("fused", M=M, K=K, N=N, ranks=ranks, max_rank=max_rank, max_loras=len(ranks) + 3,
                           none_frac=0.15, scale2=0.02, b_std=0.1, seed=M + N)
    dc = DeviceCase(cuda, atlas, case)
    y, variant = dc.run(with_ranks=with_ranks, flags=_tc(atlas))
    assert variant == atlas.VARIANT_TCGEN05
    want = ideal(oracle, case, use_ranks=with_ranks)
    assert_close(oracle, y, want, "fused")
    # B_s through the address tables (no strided pool declared) must give the same bits as B_s by TMA
    y_tab, _ = dc.run(with_ranks=with_ranks, flags=_tc(atlas), strided=False)
    assert np.array_equal(y_tab, y)
    yb, _ = dc.run(lora=False, flags=_tc(atlas))
    none = case.seq_slot < 0
    assert none.any() and np.array_equal(y[none], yb[none])            # routing is exact
    # the LoRA term is visible at this scale, and the device result tracks it
    base = ideal(oracle, case, lora=False)
    assert np.abs(want - base)[~none].mean() > 0.05
    got = oracle.bf16_to_f32(y)
    num = ((got - base)[~none] * (want - base)[~none]).sum()
    den = np.linalg.norm((got - base)[~none]) * np.linalg.norm((want - base)[~none])
    assert num / den > 0.99
    assert atlas.device_status() == 0


@pytest.mark.parametrize("M,K,N,ranks,max_rank", [
    (1, 288, 128, [8], 8),                               # one 256-wide stage and a 32-wide rest
    (16, 320, 200, [16] * 4, 16),                        # scale rows of 20 bytes: no K block of the rest is whole
    (77, 2880, 520, [16] * 8, 16),                       # split K over an odd number of K blocks
    (300, 544, 264, [8, 64], 64),                        # CTA pairs, a half K block at the end, partial second token tile
    (40, 512, 256, [128, 16, 65], 128),                  # eight granules of one slot
    (300, 1056, 384, [128] * 16, 128),                   # both at once, 128 granules per tile
    (1100, 512, 2304, [128, 72], 128),                   # token tiles of 128, ranks above 64
    (1100, 512, 4096, [128, 72], 128),                   # two-tile persistent form, ranks above 64
    (8, 8480, 256, [104], 104),                          # max_rank not a multiple of 16, long K
])
def test_shapes_beyond_the_forced_path(cuda, atlas, oracle, M, K, N, ranks, max_rank):
    """K a multiple of 32 only, ranks above 64: the default path takes them to the tensor cores, in every form a call can have,
    while what is refused there (a forced path, FP4 activations) stays refused."""
    from atlas_b200 import synth
    case = synth.make_case("wide", M=M, K=K, N=N, ranks=ranks, max_rank=max_rank, max_loras=len(ranks) + 3, none_frac=0.15,
                           scale2=0.02, b_std=0.1, seed=M + K)
    dc = DeviceCase(cuda, atlas, case, x_row_stride=K + 8, out_row_stride=N + 8)
    want = ideal(oracle, case)
    y, variant = dc.run(lora_ws=True)
    assert variant == atlas.VARIANT_TCGEN05
    assert (atlas.last_launch_shape()["persistent_tiles_per_pass"] == 2) == (N == 4096)
    assert_close(oracle, y[:, :N], want, "default path")
    assert (y[:, N:] == 0x7FC0).all()
    if K < 8192:                                         # tiles from the shrink, tiles built in the kernel, B_s by address
        for form in (dict(), dict(strided=False), dict(lora_ws=True, flags=atlas.FLAG_REUSE_SHRINK)):
            assert_close(oracle, dc.run(**form)[0][:, :N], want, f"form {form}")
    yb, variant = dc.run(lora=False)
    assert variant == atlas.VARIANT_TCGEN05
    none = case.seq_slot < 0
    assert np.array_equal(y[none][:, :N], yb[none][:, :N])      # routing is exact
    y_simt, variant = dc.run(flags=atlas.FLAG_FORCE_SIMT)
    assert variant == atlas.VARIANT_SIMT
    # no further from the FP32 result than the path that took these shapes, which rounds base and delta to BF16 before it adds
    err = [np.linalg.norm(oracle.bf16_to_f32(b[:, :N].copy()) - want) for b in (y, y_simt)]
    assert err[0] <= err[1]
    for flags in (atlas.FLAG_FORCE_TCGEN05, atlas.FLAG_ACT_FP4):
        with pytest.raises(atlas.AtlasError):
            dc.run(flags=flags, lora_ws=True)
    assert atlas.device_status() == 0


@pytest.mark.parametrize("M,K,N,ranks,max_rank", [
    (1, 256, 16, [8], 8),                                # two K steps for eight warps, one feature tile
    (5, 288, 40, [16, 8], 16),                           # K step of one thread's 32 codes, features past a tile
    (8, 1056, 5000, [24, 128, 64], 128),                 # 32 features per CTA, granule and a half
    (9, 512, 1040, [16] * 9, 16),                        # second n-tile with one token
    (16, 2304, 5008, [8, 64], 64),                       # full second n-tile, an odd number of K steps per warp
])
def test_small_batches(cuda, atlas, oracle, M, K, N, ranks, max_rank):
    """The form for up to sixteen tokens: against the oracle, with and without adapters, and a token's bits do not depend on
    the tokens beside it."""
    from atlas_b200 import synth
    case = synth.make_case("small", M=M, K=K, N=N, ranks=ranks, max_rank=max_rank, max_loras=len(ranks) + 1, none_frac=0.2 if M > 1 else 0.0,
                           scale2=0.02, b_std=0.1, seed=M + K)
    dc = DeviceCase(cuda, atlas, case, x_row_stride=K + 8, out_row_stride=N + 3)
    y, variant = dc.run()
    assert variant == atlas.VARIANT_TCGEN05 and atlas.last_launch_shape()["token_tile"] == 8
    assert_close(oracle, y[:, :N], ideal(oracle, case), "fused")
    assert (y[:, N:] == 0x7FC0).all()
    y_tab, _ = dc.run(strided=False)
    assert np.array_equal(y_tab, y)
    yb, _ = dc.run(lora=False)
    assert_close(oracle, yb[:, :N], ideal(oracle, case, lora=False), "base")
    none = case.seq_slot < 0
    assert np.array_equal(y[none], yb[none])             # (N >= 2 K where there are more than eight: both calls take this form)
    import copy
    c2 = copy.copy(case)
    c2.x, c2.seq_slot = case.x[::-1].copy(), case.seq_slot[::-1].copy()
    y2, _ = DeviceCase(cuda, atlas, c2, x_row_stride=K + 8, out_row_stride=N + 3).run()
    assert np.array_equal(y2, y[::-1])
    assert atlas.device_status() == 0


@pytest.mark.parametrize("M,K,N,ads,max_rank,small", [
    (8, 512, 264, 3, 64, True), (9, 512, 264, 3, 16, False), (9, 512, 1024, 3, 16, True),         # N >= 2 K beyond eight tokens
    (16, 512, 1024, 16, 32, True), (16, 512, 1024, 16, 40, False), (16, 512, 1024, 2, 64, True),  # up to 32 granules there
    (17, 512, 1024, 3, 16, False), (16, 512, 264, 0, 8, True),
    (6, 14336, 136, 2, 64, True), (7, 14336, 136, 2, 64, False), (7, 14336, 136, 2, 32, True), (8, 14336, 136, 2, 32, False),
])
def test_which_batches_are_small(cuda, atlas, oracle, M, K, N, ads, max_rank, small):
    """Either side of every line of the rule; what runs instead is the tcgen05 form, with the same values."""
    from atlas_b200 import synth
    case = synth.make_case("line", M=M, K=K, N=N, ranks=[max_rank] * max(ads, 1), max_rank=max_rank, scale2=0.02, b_std=0.1, seed=M + N)
    y, variant = DeviceCase(cuda, atlas, case).run(lora=ads > 0)
    assert variant == atlas.VARIANT_TCGEN05
    assert (atlas.last_launch_shape()["token_tile"] == 8) == small
    assert_close(oracle, y, ideal(oracle, case, lora=ads > 0), "either form")
    assert atlas.device_status() == 0


@pytest.mark.parametrize("M,K,N,ranks,max_rank", [
    (8, 512, 72, [16, 8, 24], 24),                       # 16 features per CTA, one n-tile
    (7, 288, 5000, [128, 16], 128),                      # 32 features per CTA, eight granules
    (16, 512, 1040, [16] * 5, 16),                       # two n-tiles
    (13, 1056, 5008, [40, 72], 72),
])
def test_small_batches_keep_adapters_apart(cuda, atlas, oracle, M, K, N, ranks, max_rank):
    """An infinity and a NaN in one adapter's B are its own rows' business."""
    from atlas_b200 import synth
    import copy
    case = synth.make_case("apart", M=M, K=K, N=N, ranks=ranks, max_rank=max_rank, max_loras=len(ranks) + 1, none_frac=0.2,
                           scale2=0.02, b_std=0.1, seed=M + N)
    case.seq_slot[:3] = [0, 1, -1]
    y_clean, _ = DeviceCase(cuda, atlas, case).run()
    bad = copy.deepcopy(case)
    bad.adapters[0].b[0, 0], bad.adapters[0].b[N - 1, ranks[0] - 1] = 0x7F80, 0x7FC0
    y, variant = DeviceCase(cuda, atlas, bad).run()
    assert variant == atlas.VARIANT_TCGEN05 and atlas.last_launch_shape()["token_tile"] == 8
    hit = case.seq_slot == 0
    assert np.array_equal(y[~hit], y_clean[~hit])
    assert np.array_equal(y[hit][:, 1:N - 1], y_clean[hit][:, 1:N - 1])
    assert not np.isfinite(oracle.bf16_to_f32(y[hit][:, [0, N - 1]].copy())).any()
    assert atlas.device_status() == 0


@pytest.mark.parametrize("M,K,N,ranks,max_rank", [
    (17, 288, 130, [16, 8, 24], 24),                     # odd row stride: no row but the first on a 16-byte boundary
    (77, 2880, 520, [16] * 8, 16),                       # split K
    (40, 512, 256, [128, 16, 65], 128),                  # ranks above 64
    (300, 1056, 384, [128] * 6, 128),                    # CTA pairs
    (1100, 512, 4096, [128, 72], 128),                   # persistent form
])
def test_shapes_beyond_the_forced_path_keep_adapters_apart(cuda, atlas, oracle, M, K, N, ranks, max_rank):
    """An infinity and a NaN in one adapter's B and a NaN in one token's x are the business of their own rows."""
    from atlas_b200 import synth
    import copy
    case = synth.make_case("apart", M=M, K=K, N=N, ranks=ranks, max_rank=max_rank, max_loras=len(ranks) + 1, none_frac=0.2,
                           scale2=0.02, b_std=0.1, seed=M + N)
    case.seq_slot[:4] = [0, 1, -1, 1]
    stride = N + 1 if M == 17 else N
    bad = copy.deepcopy(case)
    bad.adapters[0].b[1, 0], bad.adapters[0].b[N - 1, ranks[0] - 1] = 0x7F80, 0x7FC0
    bad.x[3, 5] = 0x7FC0
    for form in (dict(lora_ws=True), dict(strided=False)):
        y_clean, _ = DeviceCase(cuda, atlas, case, out_row_stride=stride).run(**form)
        y, variant = DeviceCase(cuda, atlas, bad, out_row_stride=stride).run(**form)
        assert (atlas.last_launch_shape()["persistent_cta_pairs"] > 0) == (M == 1100 and "lora_ws" in form)
        assert variant == atlas.VARIANT_TCGEN05
        hit = case.seq_slot == 0
        clean = ~hit
        clean[3] = False
        at = np.array([1, N - 1])
        rest = np.setdiff1d(np.arange(N), at)
        assert np.array_equal(y[clean][:, rest], y_clean[clean][:, rest])
        assert np.array_equal(y[hit][:, rest], y_clean[hit][:, rest])
        assert_close(oracle, y[clean][:, at], ideal(oracle, case)[clean][:, at], "computed again")
        assert not np.isfinite(oracle.bf16_to_f32(y[hit][:, at].copy())).any()
        assert not np.isfinite(oracle.bf16_to_f32(y[3:4, :N].copy())).any()
    assert atlas.device_status() == 0


@pytest.mark.parametrize("M,K,N,max_rank", [
    (8, 512, 136, 24),                                   # the smallest batches
    (40, 512, 136, 24),
    (77, 288, 200, 16),                                  # K not a multiple of 256
    (300, 512, 264, 72),                                 # CTA pairs, ranks above 64
])
def test_b_at_any_address(cuda, atlas, oracle, M, K, N, max_rank):
    """Without a strided pool B_s is read wherever its table entry says, two bytes past a 16-byte boundary too."""
    from atlas_b200 import synth
    case = synth.make_case("anywhere", M=M, K=K, N=N, ranks=[8, 16, max_rank], max_rank=max_rank, none_frac=0.1, scale2=0.02,
                           b_std=0.1, seed=M + K)
    dc = DeviceCase(cuda, atlas, case)
    want, _ = dc.run(strided=False)
    assert_close(oracle, want, ideal(oracle, case), "aligned")
    pool = dc.pool.b_pool
    moved = cuda.empty(pool.numel() + 8, dtype=pool.dtype, device="cuda")
    moved[1:1 + pool.numel()].copy_(pool.reshape(-1))
    dc.pool._b_host = [a and a - pool.data_ptr() + moved.data_ptr() + 2 for a in dc.pool._b_host]
    dc.pool.refresh_tables()
    y, variant = dc.run(strided=False)
    assert variant == atlas.VARIANT_TCGEN05
    assert np.array_equal(y, want)
    assert atlas.device_status() == 0


def test_token_permutation_is_bit_exact(cuda, atlas, oracle):
    from atlas_b200 import synth
    import copy
    case = synth.make_case("perm", M=96, K=512, N=256, ranks=[16] * 6, max_rank=16, none_frac=0.2, scale2=0.02, b_std=0.3, seed=2)
    y, _ = DeviceCase(cuda, atlas, case).run(flags=_tc(atlas))
    perm = np.random.default_rng(0).permutation(case.M)
    c2 = copy.copy(case)
    c2.x, c2.seq_slot = case.x[perm].copy(), case.seq_slot[perm].copy()
    y2, _ = DeviceCase(cuda, atlas, c2).run(flags=_tc(atlas))
    assert np.array_equal(y2, y[perm])


def test_bad_slot_is_recorded_not_fatal(cuda, atlas, oracle):
    from atlas_b200 import synth
    case = synth.make_case("bad", M=16, K=256, N=128, ranks=[8, 8], max_rank=8, max_loras=4, ids="distinct", scale2=0.02, seed=6)
    case.seq_slot[3] = 77                   # beyond the tables
    case.seq_slot[4] = 2                    # resident slot with null entries
    dc = DeviceCase(cuda, atlas, case)
    y, _ = dc.run(flags=_tc(atlas))
    yb, _ = dc.run(lora=False, flags=_tc(atlas))
    assert np.array_equal(y[3], yb[3]) and np.array_equal(y[4], yb[4])
    assert atlas.device_status() == 1
    want = ideal(oracle, case)
    assert_close(oracle, y, want, "fused with bad slots")


def test_auto_dispatch_and_fallback(cuda, atlas, oracle):
    from atlas_b200 import synth
    ok = synth.make_case("d", M=8, K=256, N=128, ranks=[8], max_rank=8, scale2=0.02, seed=1)
    _, v = DeviceCase(cuda, atlas, ok).run()
    assert v == atlas.VARIANT_TCGEN05
    odd = synth.make_case("d", M=8, K=272, N=128, ranks=[8], max_rank=8, scale2=0.02, seed=1)   # K % 256 != 0
    dc = DeviceCase(cuda, atlas, odd)
    y, v = dc.run()
    assert v == atlas.VARIANT_SIMT
    assert_close(oracle, y, ideal(oracle, odd), "fallback")
    with pytest.raises(atlas.AtlasError):
        dc.run(flags=atlas.FLAG_FORCE_TCGEN05)


def test_first_cuda_call_of_a_thread(cuda, atlas, oracle):
    """A thread that has made no call of CUDA yet: tensor maps are encoded there too."""
    import threading
    from atlas_b200 import synth
    case = synth.make_case("thread", M=40, K=512, N=136, ranks=[8], max_rank=8, scale2=0.02, seed=5)
    dc = DeviceCase(cuda, atlas, case)
    want, _ = dc.run(lora=False)
    y = cuda.zeros((40, 136), dtype=cuda.int16, device="cuda")
    d = atlas.make_linear_desc(x=dc.x, m=40, k=512, n=136, y=y, w_packed=dc.packed, w_scale=dc.scales, scale2=case.scale2)
    said = []

    def call():
        try:
            said.append(atlas.nvfp4_lora_linear(d, 0))
        except atlas.AtlasError as e:
            said.append(e)

    cuda.cuda.synchronize()
    thread = threading.Thread(target=call)
    thread.start()
    thread.join()
    cuda.cuda.synchronize()
    assert said == [atlas.VARIANT_TCGEN05]
    assert np.array_equal(y.cpu().numpy().view(np.uint16), want)


def test_more_tensor_maps_than_are_kept(cuda, atlas, oracle):
    """Two passes over more activation addresses than a thread keeps encoded maps for, from two threads at once: the same bits."""
    import threading
    from atlas_b200 import synth
    M, K, N, windows = 17, 256, 64, 4600
    case = synth.make_case("maps", M=M + windows, K=K, N=N, ranks=[8], max_rank=8, scale2=0.02, seed=4)
    dc = DeviceCase(cuda, atlas, case)
    out = cuda.zeros((4, windows, M, N), dtype=cuda.int16, device="cuda")
    cuda.cuda.synchronize()

    def passes(t):
        stream = cuda.cuda.Stream()
        for i in range(2 * windows):
            d = atlas.make_linear_desc(x=dc.x[i % windows:], m=M, k=K, n=N, y=out[2 * t + i // windows, i % windows], w_packed=dc.packed,
                                       w_scale=dc.scales, scale2=case.scale2, flags=atlas.FLAG_FORCE_TCGEN05)
            atlas.nvfp4_lora_linear(d, stream)
        stream.synchronize()

    threads = [threading.Thread(target=passes, args=(t,)) for t in range(2)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert all(cuda.equal(out[0], out[i]) for i in (1, 2, 3))
    want = ideal(oracle, case, lora=False)
    for i in (0, 2300, windows - 1):
        assert_close(oracle, out[0, i].cpu().numpy().view(np.uint16), want[i:i + M], f"window {i}")
    assert atlas.device_status() == 0


def test_config1_full_size_sampled(cuda, atlas, oracle):
    """Benchmark configuration 1 at full size (M=256, K=5120, N=17408, 16 adapters of rank 32):
    a random sample of outputs against the oracle, and exact routing on the adapter-less rows."""
    from atlas_b200 import synth
    case = synth.baseline_config(1)
    dc = DeviceCase(cuda, atlas, case)
    y, variant = dc.run()
    assert variant == atlas.VARIANT_TCGEN05
    rng = np.random.default_rng(0)
    rows = np.sort(rng.choice(case.M, 24, replace=False)).astype(np.uint32)
    cols = np.sort(rng.choice(case.N, 96, replace=False)).astype(np.uint32)
    assert_close(oracle, y[np.ix_(rows, cols)], ideal(oracle, case, rows=rows, cols=cols), "config1 sample")
    yb, _ = dc.run(lora=False)
    none = case.seq_slot < 0
    assert np.array_equal(y[none], yb[none])
    assert atlas.device_status() == 0

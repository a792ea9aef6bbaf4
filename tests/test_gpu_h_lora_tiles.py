"""LoRA activation tiles written by the shrink (scratch in `ws`) against the in-kernel build and the oracle.

Both ways put the same BF16 values into the same K-steps, so the outputs are compared bit for bit."""
import numpy as np
import pytest

from gpu_util import DeviceCase, assert_close, ideal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags_extra", ["", "fp4", "single"])
@pytest.mark.parametrize("M,K,N,ranks,max_rank,with_ranks,ids", [
    (16, 256, 128, [16] * 4, 16, True, "uniform"),
    (64, 512, 256, [8, 16, 32, 64] * 16, 64, True, "distinct"),    # every token its own adapter, mixed ranks
    (64, 512, 256, [8, 16, 32, 64] * 8, 64, False, "uniform"),     # no rank table: every slot counts max_rank
    (300, 512, 384, [32] * 16, 32, True, "uniform"),               # two token tiles, the second partial
    (130, 256, 200, [8, 24], 24, True, "uniform"),                 # max_rank not a multiple of 16
    (700, 256, 256, [16] * 40, 16, True, "zipf"),                  # three tiles, many adapters
])
def test_tiles_match_in_kernel_build(cuda, atlas, oracle, M, K, N, ranks, max_rank, with_ranks, ids, flags_extra):
    from atlas_b200 import synth
    case = synth.make_case("tiles", M=M, K=K, N=N, ranks=ranks, max_rank=max_rank, max_loras=len(ranks) + 3, ids=ids,
                           none_frac=0.15, scale2=0.02, b_std=0.1, seed=M + N + 7)
    dc = DeviceCase(cuda, atlas, case)
    fp4 = flags_extra == "fp4"
    mode = atlas.FLAG_FORCE_TCGEN05 | (atlas.FLAG_ACT_FP4 if fp4 else 0) | (atlas.FLAG_NO_CTA_PAIR if flags_extra == "single" else 0)
    y_build, _ = dc.run(with_ranks=with_ranks, flags=mode)
    dc.lora_t.zero_()                                   # the tile path must not depend on lora_t
    y_tiles, variant = dc.run(with_ranks=with_ranks, flags=mode, lora_ws=True)
    assert variant == atlas.VARIANT_TCGEN05
    assert atlas.device_status() == 0
    assert (dc.lora_t == 0).all()
    assert_close(oracle, y_tiles, ideal(oracle, case, use_ranks=with_ranks, act_fp4=fp4), "tiles")
    assert np.array_equal(y_tiles, y_build)
    # a second call (fresh scratch) gives the same bits
    y_again, _ = dc.run(with_ranks=with_ranks, flags=mode, lora_ws=True)
    assert np.array_equal(y_again, y_tiles)


def test_scratch_too_small_falls_back_to_the_build(cuda, atlas, oracle):
    from atlas_b200 import synth
    case = synth.make_case("tiles_small", M=64, K=256, N=128, ranks=[16] * 8, max_rank=16, seed=11, b_std=0.1, scale2=0.02)
    dc = DeviceCase(cuda, atlas, case)
    y0, _ = dc.run(flags=atlas.FLAG_FORCE_TCGEN05)
    y = cuda.full((64, 128), 0x7FC0, dtype=cuda.int16, device="cuda")
    ws = cuda.zeros(1024, dtype=cuda.uint8, device="cuda")
    d = atlas.make_linear_desc(x=dc.x, m=64, k=256, n=128, y=y, w_packed=dc.packed, w_scale=dc.scales, scale2=case.scale2,
                               seq_slot=dc.seq_slot, route=dc.pool.route(True, True), lora_t=dc.lora_t,
                               flags=atlas.FLAG_FORCE_TCGEN05, ws=ws, ws_bytes=1024)
    atlas.nvfp4_lora_linear(d)
    cuda.cuda.synchronize()
    assert np.array_equal(y.cpu().numpy().view(np.uint16), y0)
    assert (ws == 0).all()
    assert atlas.device_status() == 0


@pytest.mark.parametrize("M,K,N,strided_ws", [
    (8, 512, 1040, True),              # the plain call takes the form for the smallest batches and leaves no tiles
    (8, 512, 1040, False),             # ... without scratch both read rows of lora_t
    (1237, 512, 4096, True),           # the plain call's passes of two 192-token tiles fit one wave
])
def test_reuse_after_a_plain_call(cuda, atlas, oracle, M, K, N, strided_ws):
    """FLAG_REUSE_SHRINK together with a flag for comparison runs, after a call without: the bits of a call that computes its
    own shrink, whatever form the plain call left its result in."""
    from atlas_b200 import synth
    case = synth.make_case("reuse", M=M, K=K, N=N, ranks=[16] * 5, max_rank=16, max_loras=6, none_frac=0.1, scale2=0.02,
                           b_std=0.1, seed=M)
    dc = DeviceCase(cuda, atlas, case)
    y_plain, _ = dc.run(lora_ws=strided_ws)
    ws = dc.ws if strided_ws else None
    left, t_left = ws.clone() if strided_ws else None, dc.lora_t.clone()
    assert_close(oracle, y_plain, ideal(oracle, case), "plain")
    for flag in (0, atlas.FLAG_FORCE_TCGEN05, atlas.FLAG_NO_K_SPLIT, atlas.FLAG_NO_CTA_PAIR, atlas.FLAG_NO_PERSISTENT, atlas.FLAG_ONE_TILE_PASS):
        want, _ = dc.run(flags=flag, lora_ws=strided_ws)
        dc.lora_t.copy_(t_left)
        y, _ = dc.run(flags=flag | atlas.FLAG_REUSE_SHRINK, ws=left.clone() if strided_ws else None)
        assert np.array_equal(y, want), f"flag {flag}"
    assert atlas.device_status() == 0


@pytest.mark.parametrize("M,K,N,max_rank", [(9, 1024, 1024, 16), (16, 4096, 4096, 32), (12, 5120, 1280, 48)])
def test_reuse_beyond_eight_tokens(cuda, atlas, oracle, M, K, N, max_rank):
    """FLAG_REUSE_SHRINK on the small-batch kernel, N < 2 K: the rows of t that the plain call left are read, not computed again."""
    from atlas_b200 import synth
    case = synth.make_case("reuse", M=M, K=K, N=N, ranks=[max_rank, 8], max_rank=max_rank, none_frac=0.1, scale2=0.02, b_std=0.1, seed=M)
    dc = DeviceCase(cuda, atlas, case)
    plain, _ = dc.run(lora_ws=True)
    assert atlas.last_launch_shape()["token_tile"] == 8
    assert np.array_equal(dc.run(lora_ws=True, flags=atlas.FLAG_REUSE_SHRINK)[0], plain)
    dc.lora_t.zero_()
    reused, _ = dc.run(lora_ws=True, flags=atlas.FLAG_REUSE_SHRINK)
    assert np.array_equal(reused, dc.run(lora=False)[0]) and not np.array_equal(reused, plain)
    assert atlas.device_status() == 0

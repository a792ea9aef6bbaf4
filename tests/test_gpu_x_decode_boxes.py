"""The small-batch kernel with its weights by TMA (large layers, or many granules over medium ones) against the same rows as layers of
their own, small enough for the warps' loads: the same bits."""
import pytest

pytestmark = pytest.mark.gpu


# 16 and 32 features a CTA, eight and four warps, the last CTA ragged; K ends 256 and 512 into a stage, and with one
@pytest.mark.parametrize("n,k,loras,rank", [(8200, 8448, 0, 0), (16390, 4352, 0, 0), (9470, 7168, 3, 48), (4102, 4352, 8, 64), (8198, 4608, 8, 32),
                                            (16390, 4352, 8, 32), (18940, 4096, 8, 16), (19000, 4352, 2, 16)])
@pytest.mark.parametrize("m", [1, 5, 8])
def test_rows_of_a_large_layer(cuda, atlas, m, n, k, loras, rank):
    torch = cuda
    g = torch.Generator(device="cuda")
    g.manual_seed(n + k + m)
    normal = lambda *shape, std=1.0: torch.empty(shape, dtype=torch.bfloat16, device="cuda").normal_(0.0, std, generator=g)
    packed = torch.randint(0, 256, (n, k // 2), generator=g, device="cuda", dtype=torch.uint8)
    scales = torch.empty((n, k // 16), device="cuda").normal_(generator=g).abs_().to(torch.float8_e4m3fn).view(torch.uint8)
    x = normal(m, k + 8)[:, :k]
    slot = (torch.arange(m, device="cuda") % (loras + 1) - 1).to(torch.int32) if 0 < loras < m else torch.arange(m, device="cuda").to(torch.int32)
    adapters = [(normal(max(rank - 5 * s, 1), k, std=k ** -0.5), normal(n, max(rank - 5 * s, 1), std=0.05)) for s in range(loras)]
    ws = torch.full((max(atlas.lora_ws_bytes(m, max(loras, 1), max(rank, 1)), 256),), 0xA5, dtype=torch.uint8, device="cuda")
    t = torch.zeros((m, max(rank, 1)), dtype=torch.bfloat16, device="cuda")

    def call(a, b):
        y = torch.full((m, b - a), float("nan"), dtype=torch.bfloat16, device="cuda")
        kw = {}
        if loras:
            pool = atlas.LoraPool(k, b - a, rank, loras)
            for s, (aa, bb) in enumerate(adapters):
                pool.pack(s, aa, bb[a:b].contiguous(), 2.0)
            kw = dict(seq_slot=slot, route=pool.route(), lora_t=t)
        d = atlas.make_linear_desc(x=x, m=m, k=k, n=b - a, y=y, x_row_stride=k + 8, w_packed=packed[a:b], w_scale=scales[a:b], scale2=0.02,
                                   ws=ws, ws_bytes=ws.numel(), **kw)
        atlas.nvfp4_lora_linear(d)
        torch.cuda.synchronize()
        shape = atlas.last_launch_shape()
        assert shape["token_tile"] == 8 and shape["weights_by_tma"] == (b - a == n and tma)
        return y.view(torch.int16)

    # (the slices have less than 2^26 weights, or fewer than 2^24; where the batch has too few granules both sides are the warps' loads)
    tma = n * k >= 1 << 26 or min(loras, m) * ((rank + 15) // 16) >= 16
    want = torch.cat([call(a, min(a + 2048, n)) for a in range(0, n, 2048)], dim=1)
    assert torch.isfinite(want.view(torch.bfloat16)).all()
    for _ in range(3):
        assert torch.equal(call(0, n), want)
    assert atlas.device_status() == 0


@pytest.mark.parametrize("M,K,N,ads,max_rank,small", [
    (12, 1024, 1024, 2, 16, True), (16, 1056, 1100, 3, 8, True), (9, 992, 1024, 2, 16, False),       # N < 2 K from K = 1024 on
    (12, 4096, 4096, 8, 16, True), (12, 4096, 4096, 32, 64, False), (12, 5120, 1280, 2, 16, True),  # few granules, many
    (8, 1024, 1024, 8, 112, True), (8, 1024, 1024, 8, 128, False),                                  # up to eight tokens: 56 granules, 64
    (8, 14336, 6144, 2, 32, True), (8, 14336, 136, 2, 32, False), (8, 14336, 136, 8, 32, True),     # features, granules over a long K
])
def test_which_batches_below_twice_k_are_small(cuda, atlas, oracle, M, K, N, ads, max_rank, small):
    import numpy as np
    from atlas_b200 import synth
    from gpu_util import DeviceCase, assert_close, ideal
    case = synth.make_case("line", M=M, K=K, N=N, ranks=[max_rank] * ads, max_rank=max_rank, scale2=0.02, b_std=0.1, seed=M + N)
    y, variant = DeviceCase(cuda, atlas, case).run(lora_ws=True)
    assert variant == atlas.VARIANT_TCGEN05 and (atlas.last_launch_shape()["token_tile"] == 8) == small
    rows, cols = np.arange(M, dtype=np.uint32), np.sort(np.random.default_rng(N).choice(N, min(N, 96), replace=False)).astype(np.uint32)
    assert_close(oracle, y[np.ix_(rows, cols)], ideal(oracle, case, rows=rows, cols=cols), "line")
    assert atlas.device_status() == 0

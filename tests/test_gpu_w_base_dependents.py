"""Linears without adapters behind one another, each reading what the last one wrote: launched as dependents, they start while their
predecessor drains.  The same bits as with the device synchronised behind each call."""
import pytest

pytestmark = pytest.mark.gpu


# small-batch kernel, weights by the warps' loads and by TMA; one-tile kernel, its scales by TMA, from rows, and with a split K; pairs; persistent kernel (the last; FP4 too)
@pytest.mark.parametrize("m,k,fp4", [(1, 1024, False), (8, 2080, False), (16, 736, False), (1, 8192, False), (8, 8192, False), (20, 1024, False), (60, 736, False), (60, 4096, False),
                                     (250, 2048, False), (250, 2048, True), (2048, 2560, False), (2048, 2560, True)])
def test_a_chain_without_adapters(cuda, atlas, m, k, fp4):
    torch = cuda
    tma = m <= 8 and k * k >= 1 << 26
    g = torch.Generator(device="cuda")
    g.manual_seed(m + k)
    passes = 12
    weights = [torch.randint(0, 256, (k, k // 2), generator=g, device="cuda", dtype=torch.uint8) for _ in range(2)]
    scales = torch.empty((k, k // 16), device="cuda").normal_(generator=g).abs_().to(torch.float8_e4m3fn).view(torch.uint8)
    x0 = torch.empty((m, k), dtype=torch.bfloat16, device="cuda").normal_(generator=g)
    flags = atlas.FLAG_ACT_FP4 if fp4 else 0
    ws = torch.empty(atlas.act_fp4_ws_bytes(m, k) if fp4 else 256, dtype=torch.uint8, device="cuda")

    def run(sync):
        xs = [x0.clone()] + [torch.full_like(x0, float("nan")) for _ in range(passes)]
        torch.cuda.synchronize()
        for i in range(passes):
            atlas.nvfp4_lora_linear(atlas.make_linear_desc(x=xs[i], m=m, k=k, n=k, y=xs[i + 1], w_packed=weights[i % 2], w_scale=scales,
                                                           scale2=0.3 * k ** -0.5, ws=ws, ws_bytes=ws.numel(), flags=flags))
            assert atlas.last_launch_shape()["weights_by_tma"] == tma
            if sync:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return torch.stack(xs).view(torch.int16)

    want = run(True)
    assert torch.isfinite(want.view(torch.bfloat16)).all() and want[-1].count_nonzero() > m * k // 2
    for _ in range(4):
        assert torch.equal(run(False), want)
    assert atlas.device_status() == 0

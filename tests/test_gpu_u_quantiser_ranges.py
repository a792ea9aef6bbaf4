"""The quantiser's scale encoder at every rounding boundary, products too small for FP32, and the maximum over ragged sizes: bit-exact."""
import numpy as np
import pytest

from gpu_util import to_dev

pytestmark = pytest.mark.gpu


def _both(torch, atlas, oracle, w, scale2):
    N, K = w.shape
    packed = torch.zeros((N, K // 2), dtype=torch.uint8, device="cuda")
    scales = torch.zeros((N, K // 16), dtype=torch.uint8, device="cuda")
    atlas.quantize_bf16_to_nvfp4(to_dev(torch, w), packed, scales, float(np.float32(scale2)), N, K)
    torch.cuda.synchronize()
    wp, ws = oracle.quantize_bf16_to_nvfp4(w, float(np.float32(scale2)), N, K)
    assert np.array_equal(scales.cpu().numpy(), ws)
    assert np.array_equal(packed.cpu().numpy(), wp)


def test_every_magnitude_as_the_groups_maximum(cuda, atlas, oracle):
    """The maxima run over all of BF16: with tensor scales of 1/6 (1 + small steps) they meet every E4M3 value, half-way point and subnormal."""
    top = np.arange(0x7F80, dtype=np.uint16)
    w = np.zeros((len(top), 16), np.uint16)
    w[:, 5] = top | 0x8000
    w[:, 9] = top >> 1
    for scale2 in (1.0 / 6.0, np.nextafter(np.float32(1.0 / 6.0), np.float32(1)), 0.171, 1.0):
        _both(cuda, atlas, oracle, w, scale2)


@pytest.mark.parametrize("scale2", [1e-30, 1.0, 3e4, 1e30])
def test_values_far_below_the_maximum(cuda, atlas, oracle, scale2):
    """Subnormal and zero values of both signs beside large ones: products that FP32 cannot hold are zeros without a sign."""
    tops = np.arange(0x0080, 0x7F80, 0x0040, dtype=np.uint16)
    tiny = np.array([0x0000, 0x8000, 0x0001, 0x8001, 0x0002, 0x8003, 0x007F, 0x807F, 0x0080, 0x8080, 0x0100, 0x8100, 0x8F00, 0x9F00, 0xAF00], np.uint16)
    w = np.concatenate([np.tile(tiny, (len(tops), 1)), tops[:, None]], axis=1)
    _both(cuda, atlas, oracle, np.ascontiguousarray(w), scale2)


@pytest.mark.parametrize("total,offset", [(1, 0), (7, 0), (8, 0), (4097, 0), (16 * 148 * 256 * 8 * 4 + 8, 0), (1000001, 0), (4096, 1)])
def test_maximum(cuda, atlas, oracle, total, offset):
    """Fewer values than a load, a remainder behind several turns of the whole grid, an address that allows no vector loads; NaN gives way."""
    g = np.random.default_rng(total)
    w = (g.integers(0, 0x4000, total + offset).astype(np.uint16)) | (g.integers(0, 2, total + offset).astype(np.uint16) << 15)
    w[offset + total - 1] = 0xC123
    if total > 8:
        w[offset + 3] = 0x7FC0
    buf = to_dev(cuda, w)
    out = cuda.zeros(1, dtype=cuda.float32, device="cuda")
    atlas.nvfp4_global_absmax(buf[offset:], out, total)
    cuda.cuda.synchronize()
    f = (w[offset:].astype(np.uint32) << 16).view(np.float32)
    assert out.item() == np.nanmax(np.abs(f))

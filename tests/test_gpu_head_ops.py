"""Head norms and rotary positions (csrc/head_ops.cu) and the quotients by one divisor (csrc/ref_math.cuh), bit for bit against the CPU restatement."""
import numpy as np
import pytest

from util import bf16_to_f32, rand_bf16, to_dev, to_host

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def placed(a, off):
    """a device copy that starts `off` elements behind a 16-byte boundary"""
    buf = torch.zeros(a.size + 16, dtype=torch.bfloat16, device="cuda")
    t = buf[off:off + a.size].view(a.shape)
    t.copy_(to_dev(a))
    return t


def same(got, want):
    nan = np.isnan(bf16_to_f32(want))
    return np.array_equal(np.isnan(bf16_to_f32(got)), nan) and np.array_equal(got[~nan], want[~nan])


def wild(rng, a):
    """zeros of both signs, subnormals and the ends of the range among ordinary values"""
    odd = np.array([0x0000, 0x8000, 0x0001, 0x807F, 0x0080, 0x7F00, 0x1F80, 0x0D00, 0x8D80], np.uint16)
    at = rng.random(a.shape) < 0.05
    a[at] = rng.choice(odd, int(at.sum()))
    return a


@pytest.mark.parametrize("off", [0, 2])
@pytest.mark.parametrize("hd,heads,rows", [(64, 14, 1), (64, 1, 31), (64, 3, 33), (128, 12, 7), (128, 1, 65), (256, 2, 5), (256, 1, 17)])
def test_norm_and_rope(oracle, hd, heads, rows, off):
    from qwen_inference_engine_b200 import layers as L
    rng = np.random.default_rng(hd * 31 + heads * 7 + rows + off)
    x, w = rand_bf16(rng, (rows, heads * hd), 1.3), rand_bf16(rng, (hd,), 1.0)
    xd, wd = placed(x, off), placed(w, off)
    L.launch_qknorm(xd, wd, hd, rows, heads * hd, heads)
    normed = oracle.qknorm(x, w, hd, heads)
    assert np.array_equal(to_host(xd), normed)
    cos, sin = L.precompute_cos_sin(128, hd)
    cd, sd = torch.from_numpy(cos).cuda(), torch.from_numpy(sin).cuda()
    for pos in (0, 61):
        y = placed(normed[:1] if pos else normed, off)
        (L.launch_rope_single(cd, sd, y, pos, hd, heads * hd, heads) if pos else L.launch_rope(cd, sd, y, rows, hd, heads * hd, heads))
        assert np.array_equal(to_host(y), oracle.rope(cos, sin, normed[:1] if pos else normed, pos, hd, heads))


@pytest.mark.parametrize("scale", [1.0, 1e-3, 1e18])
@pytest.mark.parametrize("hd", [64, 128, 256])
def test_values_that_take_the_division(oracle, hd, scale):
    from qwen_inference_engine_b200 import layers as L
    rng = np.random.default_rng(hd)
    x, w = wild(rng, rand_bf16(rng, (40, 4 * hd), scale)), rand_bf16(rng, (4 * hd,), 1.0)
    x[0] = 0
    x[1, ::2] = 0x8000
    x[2, 5] = 0x7F80
    xd, wd = to_dev(x), to_dev(w)
    y = torch.zeros_like(xd)
    L.launch_rms(xd, wd, y, 4 * hd, 40)
    assert same(to_host(y), oracle.rmsnorm(x, w))
    L.launch_qknorm(xd, wd[:hd], hd, 40, 4 * hd, 4)
    assert same(to_host(xd), oracle.qknorm(x, w[:hd], hd, 4))


def test_every_significand_of_the_numerator(oracle):
    """one row holds every bf16 significand; the rows' divisors are spread over [1, 4)"""
    from qwen_inference_engine_b200 import layers as L
    rng = np.random.default_rng(3)
    x = np.tile((0x3F80 + np.arange(128)).astype(np.uint16), (4000, 2))
    x[:, 128:] = rand_bf16(rng, (4000, 128), 1.0)
    w = np.full(256, 0x3F80, np.uint16)
    y = torch.zeros(4000, 256, dtype=torch.bfloat16, device="cuda")
    L.launch_rms(to_dev(x), to_dev(w), y, 256, 4000)
    assert np.array_equal(to_host(y), oracle.rmsnorm(x, w))


@pytest.mark.parametrize("hd,heads,rows,off", [(64, 14, 146, 0), (64, 14, 147, 0), (64, 14, 438, 2), (64, 14, 439, 2), (128, 12, 85, 0), (128, 12, 86, 0), (128, 12, 257, 2),
                                               (256, 2, 256, 0), (256, 2, 257, 0), (256, 28, 1429, 2)])
def test_positions_around_the_rule(oracle, hd, heads, rows, off):
    """both layouts of a head, on and off a 16-byte boundary, on both sides of the number of heads that chooses between them"""
    from qwen_inference_engine_b200 import layers as L
    rng = np.random.default_rng(hd + rows)
    x = rand_bf16(rng, (rows, heads * hd), 1.3)
    cos, sin = L.precompute_cos_sin(rows, hd)
    y = placed(x, off)
    L.launch_rope(torch.from_numpy(cos).cuda(), torch.from_numpy(sin).cuda(), y, rows, hd, heads * hd, heads)
    assert np.array_equal(to_host(y), oracle.rope(cos, sin, x, 0, hd, heads))

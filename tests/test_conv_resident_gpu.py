"""The forward convolution that keeps its weights in shared memory (layers that fit, from four 16 x 16 tiles per
SM on) against the kernel that small images take. Both add the same products in the same order, so a batch that
reaches the first and its images one by one, which stay with the second, have to agree bit for bit: no tolerance.
The oracle comparison of the same kernels is in test_denoiser_gpu.py.
"""
import pytest

from sparkle_gb300 import native

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dn():
    d = native.Denoiser(0, seed=3)
    yield d
    d.close()


def batch_for(h: int, w: int) -> int:
    """Images of h x w that give at least four and a bit 16 x 16 tiles per SM, an odd number of them."""
    tiles = -(-h // 16) * -(-w // 16)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return (4 * sms // tiles + 1) | 1


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("cin,cout", [(32, 32), (96, 32), (32, 64), (64, 64), (160, 32)])
@pytest.mark.parametrize("h,w", [(96, 112), (33, 47), (17, 9), (128, 16)])
def test_batch_matches_single_images(dn, h, w, cin, cout, masked):
    n = batch_for(h, w)
    gen = torch.Generator(device="cuda").manual_seed(h * 1000 + w + cin + cout)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=gen).to(torch.bfloat16)
    # Channel slices of wider buffers on both sides: pixel strides of their own, neighbours left alone.
    x, wt, mask = rand(n, h, w, cin + 32), rand(cout, 9, cin) * 0.1, rand(n, h, w, cout)
    bias = torch.randn(cout, device="cuda", generator=gen)
    y = torch.full((n, h, w, cout + 32), 7.0, device="cuda", dtype=torch.bfloat16)
    one = y.clone()
    kw = dict(x_ld=cin + 32, y_ld=cout + 32)
    opts = lambda i: dict(kw, mask=mask[i:], mask_ld=cout) if masked else dict(kw, bias=bias, relu=True)
    dn.conv3x3(0, x[..., 8:], cin, wt, y[..., 16:], cout, n, h, w, **opts(0))
    for i in range(n):
        dn.conv3x3(0, x[i:, ..., 8:], cin, wt, one[i:, ..., 16:], cout, 1, h, w, **opts(i))
    assert torch.equal(y, one)
    assert torch.all(y[..., :16] == 7.0) and torch.all(y[..., 16 + cout:] == 7.0)


@pytest.mark.parametrize("h,w", [(128, 128), (100, 72)])
def test_network_batch_matches_single_images(dn, h, w):
    """The whole network, with its pooled layers and skip slices."""
    n = batch_for(h, w)
    gen = torch.Generator(device="cuda").manual_seed(5)
    feats = torch.rand(n, h, w, 10, device="cuda", generator=gen)
    batch = dn.infer(feats).clone()
    for i in range(n):
        assert torch.equal(batch[i], dn.infer(feats[i:i + 1].contiguous())[0])


@pytest.mark.parametrize("cin,cout", [(32, 96), (128, 128), (224, 96), (32, 256)])
@pytest.mark.parametrize("waves,extra", [(1, 0), (1, 1), (2, 0), (2, 1)])
def test_ring_depths_agree(dn, cin, cout, waves, extra):
    """Wide layers on grids of one and two CTAs per SM and just above: the ring's depth changes there, the sums
    do not. One tile of 16 x 8 pixels per image."""
    n = waves * torch.cuda.get_device_properties(0).multi_processor_count + extra
    gen = torch.Generator(device="cuda").manual_seed(cin + cout + n)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=gen).to(torch.bfloat16)
    x, wt, bias = rand(n, 8, 16, cin), rand(cout, 9, cin) * 0.1, torch.randn(cout, device="cuda", generator=gen)
    y = torch.zeros(n, 8, 16, cout, device="cuda", dtype=torch.bfloat16)
    one = y.clone()
    dn.conv3x3(0, x, cin, wt, y, cout, n, 8, 16, bias=bias, relu=True)
    for i in (0, 1, n // 2, n - 1):
        dn.conv3x3(0, x[i:], cin, wt, one[i:], cout, 1, 8, 16, bias=bias, relu=True)
        assert torch.equal(y[i], one[i])

"""The 3x3 convolution's TMA path at the edges of its tiles, against the gather
kernel (layout 2).  Tiles of 128 pixels add the same products in the same order
as the gather kernel: equal bits.  Bands of rows (32 or 64 output channels,
widths that are multiples of 128) add them in another order: both are FP32 sums
rounded to bf16, which differ in a few last places (2^-8 each)."""
import pytest

from test_gpu_unet import conv_ref, run_conv

pytestmark = pytest.mark.gpu

TILES = [
    # (cin, cout, (n, h, w)): 64- and 32-channel chunks, tiles of 128 x 1 to 8 x 16 pixels,
    # ragged right and lower edges, one tile and more tiles than SMs
    (32, 32, (1, 1, 1)), (64, 32, (2, 5, 7)), (32, 64, (1, 23, 23)), (64, 64, (3, 46, 46)),
    (96, 64, (1, 17, 200)), (32, 32, (1, 3, 128)), (64, 32, (1, 6, 130)), (64, 64, (1, 3, 256)),
    (64, 128, (1, 32, 32)), (128, 128, (5, 96, 96)), (32, 128, (2, 16, 16)), (128, 128, (2, 33, 65)),
    (128, 256, (1, 12, 20)), (256, 256, (16, 40, 48)), (96, 256, (1, 2, 128)),
]
BANDS = [
    (32, 32, (1, 4, 128)), (64, 32, (2, 8, 256)), (96, 32, (1, 12, 128)), (64, 32, (16, 64, 384)),
    (32, 64, (1, 2, 128)), (64, 64, (1, 4, 256)), (128, 64, (3, 6, 128)), (64, 64, (16, 50, 384)),
]


def data(cin, cout, shape):
    import torch

    torch.manual_seed(cin + cout + shape[1])
    x = torch.randn(*shape, cin, device="cuda").bfloat16()
    w = (torch.randn(cout, 9, cin, device="cuda") / (3 * cin ** 0.5)).bfloat16()
    return x, w, torch.randn(cout, device="cuda") * 0.1


@pytest.mark.parametrize("cin,cout,shape", TILES)
def test_tiles_equal_the_gather_kernel(gb, cin, cout, shape):
    import torch

    x, w, b = data(cin, cout, shape)
    for relu in (True, False):
        assert torch.equal(run_conv(gb, x, w, b, relu, 0), run_conv(gb, x, w, b, relu, 2))


@pytest.mark.parametrize("cin,cout,shape", BANDS)
def test_bands_near_the_gather_kernel(gb, cin, cout, shape):
    x, w, b = data(cin, cout, shape)
    ref = conv_ref(x, w, b, relu=True)
    y, y2 = run_conv(gb, x, w, b, True, 0).float(), run_conv(gb, x, w, b, True, 2).float()
    assert float((y - y2).norm() / ref.norm()) < 1e-3
    assert float((y - ref).abs().max()) < 2 ** -7 * float(ref.abs().max())

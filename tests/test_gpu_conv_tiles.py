"""The 3x3 convolution at the edges of its tiles: image rows that do not fill a
tile of four or two rows, widths around one and two tiles of 128 pixels, more
tiles than resident blocks, one pixel, and the layers on either side of the line
between resident weights and the load ring.  Bounds: those of the convolution
tests (BF16 rounding of the output).  Inputs off a 16-byte boundary are refused
before anything is launched."""
import pytest

from test_gpu_warmstart import _close, _ref_conv

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,H,W,c0,c1,N", [
    (1, 1, 1, 16, 0, 16), (2, 3, 127, 16, 0, 16), (1, 5, 129, 32, 16, 16), (1, 4, 256, 32, 0, 32),
    (3, 7, 257, 32, 0, 64), (40, 61, 130, 16, 0, 16),    # 1280 tiles of four rows
    (1, 6, 131, 64, 0, 32), (1, 3, 128, 64, 0, 64), (1, 9, 70, 64, 32, 32)])
def test_conv_at_tile_edges(n, H, W, c0, c1, N):
    from feilab_b200 import warmstart
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn((n, H, W, c0), generator=g, device="cuda").to(torch.bfloat16)
    x1 = torch.randn((n, H, W, c1), generator=g, device="cuda").to(torch.bfloat16) if c1 else None
    w = (torch.randn((9, N, c0 + c1), generator=g, device="cuda") / (9 * (c0 + c1)) ** 0.5).to(torch.bfloat16)
    out = warmstart.conv3x3(x, w, None, False, in1=x1)
    torch.cuda.synchronize()
    assert warmstart.device_error() == 0
    _close(out, _ref_conv(x, x1, w, None, False))


@pytest.mark.parametrize("c0,N", [(16, 16), (64, 64)])
def test_conv_refuses_misaligned_images(c0, N):
    from feilab_b200 import warmstart
    from feilab_b200.icon import IconError
    buf = torch.zeros(2 * 128 * c0 + 8, dtype=torch.bfloat16, device="cuda")
    w = torch.zeros((9, N, c0), dtype=torch.bfloat16, device="cuda")
    with pytest.raises(IconError):
        warmstart.conv3x3(buf[1:1 + 2 * 128 * c0].view(1, 2, 128, c0), w)

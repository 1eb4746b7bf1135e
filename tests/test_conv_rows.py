"""The warp-specialised convolutions -- over rows of 128 pixels (layers whose
weights fit in shared memory, W from 128 on) and tile by tile (64 input
channels at a time) -- against the thread-gathered convolution: the same
products in the same order, so the outputs are equal bit for bit.  Shapes: one
row per CTA and fewer rows than SMs, runs that cross strips and images, one row
images, every output width and every box width, tiles of several image rows, a
grid with and without a second wave and in slices of 64 and 128 channels, fp32
and bf16 outputs, strided outputs (a slice of a wider tensor), and with and
without bias and ReLU."""
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 128, 16, 16), (1, 5, 128, 32, 32), (3, 37, 128, 32, 48), (2, 64, 256, 64, 64), (1, 211, 384, 96, 32),
          (2, 33, 256, 32, 96), (1, 300, 128, 64, 128), (1, 64, 1024, 16, 32), (5, 67, 128, 48, 64),
          (1, 32, 256, 32, 128),
          # ragged last strips: one pixel short, one over a strip and a half, rows too narrow for strips
          (1, 40, 255, 32, 32), (2, 21, 193, 16, 64), (1, 70, 344, 64, 64), (3, 5, 1000, 96, 32), (1, 9, 129, 32, 48),
          # tile by tile: rows of 64, 32, 16 pixels; many and few tiles
          (1, 16, 64, 64, 64), (2, 32, 32, 128, 256), (4, 16, 16, 384, 128), (1, 130, 128, 256, 192),
          (2, 128, 128, 128, 128), (1, 64, 128, 256, 256), (3, 64, 128, 192, 64),
          # ragged tiles: last rows, last columns, rows of 43, 100 and 7 pixels
          (1, 65, 43, 256, 128), (2, 31, 100, 128, 64), (1, 50, 7, 64, 192), (2, 9, 172, 384, 128), (1, 33, 316, 192, 64)]


@pytest.mark.parametrize("f32,relu", [(False, True), (True, False)])
@pytest.mark.parametrize("B,H,W,cin,N", SHAPES)
def test_rows_equal_gathered(B, H, W, cin, N, f32, relu):
    import torch
    from xbeach_gpu_b200 import surrogate as sg
    g = torch.Generator(device="cuda").manual_seed(B * H + W + cin + N)
    L = sg.lib()
    P, Kp = B * H * W, (9 * cin + 63) // 64 * 64
    x = torch.randn(P, cin, device="cuda", generator=g).to(torch.bfloat16)
    w = torch.zeros(N, Kp, device="cuda")
    w[:, :9 * cin] = torch.randn(N, 9 * cin, device="cuda", generator=g) / (9 * cin) ** 0.5
    w = w.to(torch.bfloat16)
    bias = torch.randn(N, device="cuda", generator=g) if relu else None
    dt = torch.float32 if f32 else torch.bfloat16
    ys = []
    for on in (0, 1):
        wide = torch.full((P, N + 16), 7.0, device="cuda", dtype=dt)
        y = wide[:, 8:8 + N] if not f32 else wide[:, :N]
        assert L.xbg_nn_conv_set_tma(on) == 0
        try:
            err = sg.conv3x3(x, w, y, B, H, W, cin, bias=bias, relu=relu)
            torch.cuda.synchronize()
        finally:
            L.xbg_nn_conv_set_tma(1)
        assert int(err.item()) == 0
        ys.append(wide)
    assert torch.equal(ys[0], ys[1])

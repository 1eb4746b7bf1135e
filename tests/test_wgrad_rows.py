"""The weight gradient with box copies (W a multiple of 64, input channels a multiple
of 16, at most 128 output channels) against the thread-gathered kernel: the same
slices in the same order, so the results are equal bit for bit; and against a
float64 im2col product of the same bf16 values, to the bound of the
thread-gathered kernel's test (1e-4 of the largest gradient).  Shapes: one image
row, one to several chunks per image row, runs that cross images, slices
without a chunk, both box widths, every output width, strided inputs, and runs
and rows for which the thread-gathered kernel stays."""
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 64, 16, 16, 1), (1, 3, 64, 32, 32, 1), (2, 5, 128, 16, 48, 3), (3, 7, 192, 48, 64, 5),
          (1, 40, 64, 64, 96, 9), (2, 33, 128, 96, 32, 16), (1, 64, 192, 32, 128, 20), (4, 16, 64, 192, 128, 12),
          (1, 9, 256, 32, 16, 2), (2, 50, 256, 16, 32, 40), (3, 11, 64, 32, 64, 16), (1, 64, 256, 64, 64, 7),
          (1, 17, 320, 32, 128, 3), (1, 20, 640, 16, 16, 6), (2, 8, 1024, 32, 32, 3), (1, 30, 100, 32, 32, 4)]


@pytest.mark.parametrize("B,H,W,cin,N,ks", SHAPES)
def test_wgrad_rows(B, H, W, cin, N, ks):
    import torch
    import torch.nn.functional as F
    from xbeach_gpu_b200 import surrogate as sg
    L = sg.lib()
    g = torch.Generator(device="cuda").manual_seed(B + 3 * H + 5 * W + cin + N + ks)
    P, Kp = B * H * W, (9 * cin + 63) // 64 * 64
    x = torch.randn(P, cin + 16, device="cuda", generator=g).bfloat16()[:, 8:8 + cin]
    dz = torch.randn(P, N + 8, device="cuda", generator=g).bfloat16()[:, :N]
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = []
    for on in (1, 1, 0):
        gw, gb = torch.full((N, Kp), 3.0, device="cuda"), torch.zeros(N, device="cuda")
        work = torch.full((L.xbg_nn_conv3x3_wgrad_work(cin, N, ks),), float("nan"), device="cuda")
        assert L.xbg_nn_conv_set_tma(on) == 0
        try:
            sg.conv3x3_wgrad(x, dz, gw, gb, work, B, H, W, cin, ks, err, accumulate=False)
            torch.cuda.synchronize()
        finally:
            L.xbg_nn_conv_set_tma(1)
        out.append((gw, gb))
    assert int(err.item()) == 0
    xi = x.double().reshape(B, H, W, cin).permute(0, 3, 1, 2)
    col = F.unfold(xi, 3, padding=1).view(B, cin, 9, H * W).permute(0, 3, 2, 1).reshape(P, 9 * cin)
    rw, rb = dz.double().t() @ col, dz.double().sum(0)
    for gw, gb in out:
        assert torch.all(gw[:, 9 * cin:] == 3.0)
        assert (gw[:, :9 * cin] - rw).abs().max() <= 1e-4 * rw.abs().max()
        assert (gb - rb).abs().max() <= 1e-4 * rb.abs().max()
    for gw, gb in out[1:]:
        assert torch.equal(out[0][0], gw) and torch.equal(out[0][1], gb)

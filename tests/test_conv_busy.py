"""The convolution and the weight gradient where every SM has work and each block
many rows (more than stages and accumulator slots hold), several launches in a row,
against the thread-gathered kernels, bit for bit: output widths whose blocks ask for
all tensor memory columns, and the widths that are left to the other kernels."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,N", [(16, 48), (16, 64), (16, 96), (16, 128), (48, 48), (32, 96), (32, 128), (64, 128)])
def test_conv_all_sms(cin, N):
    _conv(4, 256, 256, cin, N)


# runs of rows that end with their strip and runs that cross into the next one (the
# last of a strip shorter, one row longer than the rows divide, more strips than SMs),
# ragged strips, 16-channel boxes at the smallest size that takes them and below, and
# tiles either side of one block per SM in slices of 64 and of 128 channels
@pytest.mark.parametrize("B,H,W,cin,N", [(1, 256, 256, 16, 32), (1, 224, 224, 16, 32), (1, 400, 400, 16, 16),
                                         (2, 250, 300, 48, 48), (1, 304, 300, 96, 32), (1, 160, 176, 32, 32),
                                         (1, 208, 256, 64, 128), (4, 240, 254, 32, 64), (150, 3, 128, 64, 64),
                                         (1, 74, 128, 128, 128), (1, 75, 128, 128, 128), (1, 149, 128, 128, 128)])
def test_conv_runs(B, H, W, cin, N):
    _conv(B, H, W, cin, N)


# blocks whose stores take as long as their products, so that the product warp waits for accumulators
@pytest.mark.parametrize("B,H,W,cin,N", [(5, 64, 455, 64, 128), (4, 256, 256, 32, 128), (3, 194, 513, 32, 96),
                                         (5, 117, 512, 32, 64)])
def test_conv_stores_bound(B, H, W, cin, N):
    import torch
    _conv(B, H, W, cin, N, torch.float32)


def _conv(B, H, W, cin, N, out=None):
    import torch
    from xbeach_gpu_b200 import surrogate as sg
    g = torch.Generator(device="cuda").manual_seed(cin + N)
    L = sg.lib()
    P, Kp = B * H * W, (9 * cin + 63) // 64 * 64
    x = torch.randn(P, cin, device="cuda", generator=g).to(torch.bfloat16)
    w = torch.zeros(N, Kp, device="cuda")
    w[:, :9 * cin] = torch.randn(N, 9 * cin, device="cuda", generator=g) / (9 * cin) ** 0.5
    w = w.to(torch.bfloat16)
    y = [torch.zeros(P, N, device="cuda", dtype=out or torch.bfloat16) for _ in range(2)]
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    for on in (0, 1):
        assert L.xbg_nn_conv_set_tma(on) == 0
        try:
            for _ in range(1 + 9 * on):
                sg.conv3x3(x, w, y[on], B, H, W, cin, err=err)
            torch.cuda.synchronize()
        finally:
            L.xbg_nn_conv_set_tma(1)
    assert int(err.item()) == 0
    assert torch.equal(y[0], y[1])


@pytest.mark.parametrize("cin,N,W", [(16, 96, 64), (48, 96, 64), (16, 128, 64), (16, 96, 128)])
def test_wgrad_all_sms(cin, N, W):
    import torch
    from xbeach_gpu_b200 import surrogate as sg
    B, H, ks = 4, 512, 64
    g = torch.Generator(device="cuda").manual_seed(cin + N + W)
    L = sg.lib()
    P, Kp = B * H * W, (9 * cin + 63) // 64 * 64
    x = torch.randn(P, cin, device="cuda", generator=g).bfloat16()
    dz = torch.randn(P, N, device="cuda", generator=g).bfloat16()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = []
    for on in (0, 1):
        gw, gb = torch.zeros(N, Kp, device="cuda"), torch.zeros(N, device="cuda")
        work = torch.empty(L.xbg_nn_conv3x3_wgrad_work(cin, N, ks), device="cuda")
        assert L.xbg_nn_conv_set_tma(on) == 0
        try:
            for _ in range(1 + 9 * on):
                sg.conv3x3_wgrad(x, dz, gw, gb, work, B, H, W, cin, ks, err, accumulate=False)
            torch.cuda.synchronize()
        finally:
            L.xbg_nn_conv_set_tma(1)
        out.append((gw, gb))
    assert int(err.item()) == 0
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])

"""The surrogate's poolings, upsamplings and channel copies against plain torch in
the same order of fp32 operations, so equal bit for bit: one pixel, rows shorter
than a warp, ragged rows, rows of several blocks, slices of a wider tensor."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,h,w,C,ld,c0", [(1, 1, 1, 8, 8, 0), (2, 3, 5, 24, 40, 8), (1, 7, 129, 64, 96, 32),
                                           (3, 2, 33, 256, 384, 128), (1, 5, 1500, 32, 48, 0)])
def test_resample_and_copy(B, h, w, C, ld, c0):
    import torch
    from xbeach_gpu_b200 import surrogate as sg
    L, p = sg.lib(), sg._p
    sg._bind_ops(L)
    g = torch.Generator(device="cuda").manual_seed(B + h + w + C)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()   # noqa: E731
    kids = lambda t: [t[:, a::2, b::2] for a in (0, 1) for b in (0, 1)]       # noqa: E731
    lo, hi, wide = rnd(B, h, w, C), rnd(B, 2 * h, 2 * w, C), rnd(B, 2 * h, 2 * w, ld)
    sl = slice(c0, c0 + C)

    y = wide.clone()
    assert L.xbg_nn_up2(p(lo), p(y), B, h, w, C, ld, c0, None) == 0
    r = wide.clone()
    for k in kids(r):
        k[..., sl] = lo
    assert torch.equal(y, r)

    y = torch.empty_like(lo)
    assert L.xbg_nn_up2_bwd(p(wide), p(y), B, h, w, C, ld, c0, None) == 0
    a, b, c, d = (k[..., sl].float() for k in kids(wide))
    assert torch.equal(y, (((a + b) + c) + d).bfloat16())

    y = torch.empty_like(lo)
    assert L.xbg_nn_pool2(p(hi), p(y), B, 2 * h, 2 * w, C, None) == 0
    a, b, c, d = (k.float() for k in kids(hi))
    assert torch.equal(y, ((((a + b) + c) + d) * 0.25).bfloat16())

    for acc in (0, 1):
        y, r = hi.clone(), hi.clone()
        assert L.xbg_nn_pool2_bwd(p(lo), p(y), B, 2 * h, 2 * w, C, acc, None) == 0
        for k in kids(r):
            k.copy_((lo.float() * 0.25 + (k.float() if acc else 0.0)).bfloat16())
        assert torch.equal(y, r)

    P = B * 4 * h * w
    y, r = wide.clone(), wide.clone()
    assert L.xbg_nn_chan_copy(p(hi), p(y), P, C, ld, c0, 0, 0, None) == 0
    r[..., sl] = hi
    assert torch.equal(y, r)
    for acc in (0, 1):
        y = hi.clone()
        assert L.xbg_nn_chan_copy(p(y), p(wide), P, C, ld, c0, 1, acc, None) == 0
        assert torch.equal(y, (wide[..., sl].float() + (hi.float() if acc else 0.0)).bfloat16())

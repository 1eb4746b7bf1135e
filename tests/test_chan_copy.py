"""Channel copies with one and with four 16-byte pieces per thread, at the sizes where
the one takes over from the other and at the smallest, against slices: equal bit for
bit (the sum of two bf16 values is rounded once)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,C", [(1, 8), (3, 40), (149_999, 8), (150_000, 8), (149_999 // 3, 24), (50_001, 24),
                                 (899_999, 8), (900_000, 8), (300_001, 24), (257, 256)])
def test_chan_copy(P, C):
    import torch
    from xbeach_gpu_b200 import surrogate as sg
    L = sg.lib()
    sg._bind_ops(L)
    g = torch.Generator(device="cuda").manual_seed(P + C)
    ld, c0 = C + 24, 16
    x = torch.randn(P, C, device="cuda", generator=g).bfloat16()
    y = torch.randn(P, ld, device="cuda", generator=g).bfloat16()
    want = y.clone()
    want[:, c0:c0 + C] = x
    got = y.clone()
    assert L.xbg_nn_chan_copy(sg._p(x), sg._p(got), P, C, ld, c0, 0, 0, None) == 0
    for acc in (0, 1):
        back = x.clone()
        assert L.xbg_nn_chan_copy(sg._p(back), sg._p(y), P, C, ld, c0, 1, acc, None) == 0
        s = y[:, c0:c0 + C]
        assert torch.equal(back, (x.float() + s.float()).bfloat16() if acc else s)
    assert torch.equal(got, want)

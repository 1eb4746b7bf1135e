"""The updates of several arrays in one launch against one launch per array: equal
bit for bit, with arrays of one element, of whole and of ragged blocks, and none."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[1], [256, 257, 16, 70001], [0, 5, 0, 1024], [33] * 32, []])
def test_adam_many(sizes):
    import torch
    from xbeach_gpu_b200 import surrogate as sg
    L = sg.lib()
    sg._bind_ops(L)
    g = torch.Generator(device="cuda").manual_seed(len(sizes))

    def arrays():
        return [[torch.randn(n, device="cuda", generator=g), torch.zeros(n, device="cuda", dtype=torch.bfloat16),
                 *(torch.rand(n, device="cuda", generator=g) for _ in range(3))] for n in sizes if n]
    a = arrays()
    b = [[t.clone() for t in r] for r in a]
    rows = [(*(t.data_ptr() for t in r), r[0].numel()) for r in a]
    assert L.xbg_nn_adam_many((sg._AdamArray * max(1, len(rows)))(*rows), len(rows), 1e-3, 0.9, 0.999, 1e-8, 3,
                              None) == 0
    for r in b:
        assert L.xbg_nn_adam(*(sg._p(t) for t in r), r[0].numel(), 1e-3, 0.9, 0.999, 1e-8, 3, None) == 0
    torch.cuda.synchronize()
    for r, q in zip(a, b):
        assert all(torch.equal(s, t) for s, t in zip(r, q))
    assert L.xbg_nn_adam_many((sg._AdamArray * 33)(), 33, 1e-3, 0.9, 0.999, 1e-8, 3, None) != 0


def test_flip_many():
    import torch
    from xbeach_gpu_b200 import surrogate as sg
    L = sg.lib()
    sg._bind_ops(L)
    shapes = [(16, 32, 192, 320), (32, 16, 320, 192), (384, 128, 3456, 1152)]   # cin, cd, ldw, ldf
    w = [torch.randn(cd, ldw, device="cuda").bfloat16() for _, cd, ldw, _ in shapes]
    one, many = ([torch.full((cin, ldf), 9.0, device="cuda", dtype=torch.bfloat16) for cin, _, _, ldf in shapes]
                 for _ in range(2))
    rows = [(x.data_ptr(), y.data_ptr(), ldw, cin, cd, ldf) for x, y, (cin, cd, ldw, ldf) in zip(w, many, shapes)]
    assert L.xbg_nn_conv3x3_flip_many((sg._FlipLayer * 3)(*rows), 3, None) == 0
    for x, y, (cin, cd, ldw, ldf) in zip(w, one, shapes):
        assert L.xbg_nn_conv3x3_flip(sg._p(x), ldw, cin, cd, sg._p(y), ldf, None) == 0
    torch.cuda.synchronize()
    assert all(torch.equal(x, y) for x, y in zip(one, many))

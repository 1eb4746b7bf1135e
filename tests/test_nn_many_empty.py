"""Arrays without elements in the update of several arrays: at the start, between
others, in a row and at the end, and all of them; the others equal to one launch per
array bit for bit, and a byte beyond an empty array untouched."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[0, 5], [5, 0], [0, 5, 0, 1024], [256, 0, 0, 257, 0], [0, 0, 0], [0] * 31 + [3]])
def test_adam_many_empty_arrays(sizes):
    import torch
    from xbeach_gpu_b200 import surrogate as sg
    L = sg.lib()
    sg._bind_ops(L)
    g = torch.Generator(device="cuda").manual_seed(sum(sizes) + len(sizes))

    def arrays():
        return [[torch.randn(max(n, 1), device="cuda", generator=g),
                 torch.zeros(max(n, 1), device="cuda", dtype=torch.bfloat16),
                 *(torch.rand(max(n, 1), device="cuda", generator=g) for _ in range(3))] for n in sizes]
    a = arrays()
    b = [[t.clone() for t in r] for r in a]
    rows = [(*(t.data_ptr() for t in r), n) for r, n in zip(a, sizes)]
    assert L.xbg_nn_adam_many((sg._AdamArray * len(rows))(*rows), len(rows), 1e-3, 0.9, 0.999, 1e-8, 3, None) == 0
    for r, n in zip(b, sizes):
        assert L.xbg_nn_adam(*(sg._p(t) for t in r), n, 1e-3, 0.9, 0.999, 1e-8, 3, None) == 0
    torch.cuda.synchronize()
    for r, q in zip(a, b):
        assert all(torch.equal(s, t) for s, t in zip(r, q))

"""A rounding for which the grid Cholesky QR's workspace (Q rows, partial Gram
matrices: ~4 GB here) does not fit beside the train: the Householder tree takes
the bonds, with the result it gives on its own."""
import numpy as np
import pytest

import paratt_b200 as P
from paratt_b200 import Context

pytestmark = pytest.mark.gpu


def test_little_memory_left():
    torch = pytest.importorskip("torch")
    n, r = 12000, 80
    gen = torch.Generator(device="cuda").manual_seed(3)
    shape = [(r, 90, 1), (r, n, r), (1, 90, r)]
    cores = [torch.randn(s, dtype=torch.float64, device="cuda", generator=gen) / s[2] ** 0.5 for s in shape]
    ranks = [1, r, r, 1]
    outs = []
    for hog in (False, True):
        c = Context(0)
        x = P.TT(c, [90, n, 90], ranks)
        torch.cuda.synchronize()
        x.set_device(ranks, [t.data_ptr() for t in cores])
        held = None
        if hog:
            free = torch.cuda.mem_get_info()[0]
            held = torch.empty(free - (3 << 30), dtype=torch.uint8, device="cuda")
        else:
            c.cholqr(False)
        x.round(1e-10, 60)
        outs.append(x.get())
        x.close()
        c.close()
        del held
        torch.cuda.empty_cache()
    assert [t.shape for t in outs[0]] == [t.shape for t in outs[1]]
    for a, b in zip(*outs):
        assert np.array_equal(a, b)

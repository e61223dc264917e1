"""The block product takes operands and results on any 8-byte boundary.

Results that start on a 16-byte boundary are stored two elements at a time,
others one at a time: the tensor-core product gives the same bits either way.
The FP64 product takes another kernel there, whose sums run in another order:
of a few hundred terms of order 1/k, 1e-13 of the largest result is above
their rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [[64], [130, 65], [512, 200]])
@pytest.mark.parametrize("tensor", [False, True])
def test_products_on_8_byte_boundaries(v2g, dims, tensor):
    import torch

    pads = [(d + 63) // 64 * 64 for d in dims]
    total = sum(p * p for p in pads)
    rng = np.random.default_rng(len(dims))
    host = []
    for _ in range(2):
        m = np.zeros(total)
        o = 0
        for d, p in zip(dims, pads):
            m[o:o + p * p].reshape(p, p)[:d, :d] = rng.standard_normal((d, d)) / np.sqrt(d)
            o += p * p
        host.append(m)
    weights = rng.standard_normal(sum(pads))

    def product(shift):
        def put(h):
            t = torch.empty(h.size + 1, dtype=torch.float64, device="cuda")[shift:shift + h.size]
            t.copy_(torch.from_numpy(h))
            return t

        a, b, d, c = put(host[0]), put(host[1]), put(weights), put(np.full(total, np.nan))
        assert c.data_ptr() % 16 == 8 * shift
        v2g.block_gemm_device(dims, a.data_ptr(), b.data_ptr(), c.data_ptr(), d_d=d.data_ptr(), tensor_cores=tensor)
        return c.cpu().numpy()

    want, got = product(0), product(1)
    assert np.isfinite(want).all()
    if tensor:
        assert np.array_equal(want, got)
    else:
        assert np.abs(want - got).max() <= 1e-13 * np.abs(want).max()

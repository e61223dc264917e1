"""The FP64 block product's forms against numpy: split-K clusters (few tiles), FP64
tensor instructions (many), and plain loads where a buffer is not 16-byte aligned.

FP64 sums of at most 448 products of order one: 1e-12 of the largest entry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FEW, MANY = [65, 100], [65, 100, 169, 200, 64, 338, 1, 448, 400]


@pytest.mark.parametrize("dims", [FEW, MANY], ids=["few", "many"])
@pytest.mark.parametrize("ta", [False, True])
@pytest.mark.parametrize("tb", [False, True])
@pytest.mark.parametrize("scaled,offset", [(False, 0), (True, 0), (True, 1)])
def test_fp64_block_gemm_forms(v2g, dims, ta, tb, scaled, offset):
    import torch

    rng = np.random.default_rng(len(dims) + 2 * ta + tb)
    pad = [(d + 63) // 64 * 64 for d in dims]
    A, B = ([np.zeros((p, p)) for p in pad] for _ in range(2))
    D = [np.zeros(p) for p in pad]
    for d, a, b, w in zip(dims, A, B, D):
        a[:d, :d], b[:d, :d], w[:d] = rng.standard_normal((d, d)), rng.standard_normal((d, d)), rng.uniform(-1, 2, d)

    def device(blocks):
        flat = np.concatenate([np.zeros(offset)] + [m.reshape(-1) for m in blocks])
        return torch.from_numpy(flat).cuda()

    dA, dB, dD = device(A), device(B), device(D)
    dC = torch.full_like(dA, float("nan"))
    at = lambda t: t.data_ptr() + 8 * offset  # noqa: E731
    v2g.block_gemm_device(dims, at(dA), at(dB), at(dC), trans_a=ta, trans_b=tb, d_d=at(dD) if scaled else None,
                          tensor_cores=False)
    got = dC.cpu().numpy()[offset:]
    o = 0
    for p, a, b, w in zip(pad, A, B, D):
        want = ((a.T if ta else a) * (w if scaled else 1.0)) @ (b.T if tb else b)
        c = got[o:o + p * p].reshape(p, p)
        assert np.abs(c - want).max() <= 1e-12 * max(1.0, np.abs(want).max())
        o += p * p

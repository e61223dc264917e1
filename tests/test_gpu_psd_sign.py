"""The projection x = U+ / mu, z = U- on crafted blocks against numpy's eigh.

With y = 0 and c = 0 a block's U is mu x, so x sets it freely: every spectrum
that makes the sign iteration work hard (zero, rank one, clusters, eigenvalues
down to rounding, definite blocks, extreme scales) at block sizes that fill and
do not fill the 8 x 8 (or 64 x 64) tiles.  The iteration stops when
|U (1 - X^2)|_F <= 1e-15 sqrt(N) |U|_F, and its products round at
eps sqrt(N) |U|_F each; 2e-14 |U|_F per block leaves room for both.  x and z have
to be positive semidefinite to the same tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spectra(rng, n):
    yield np.zeros(n)
    yield np.ones(n) * 3.0
    yield -np.abs(rng.standard_normal(n))
    yield np.r_[2.0, np.zeros(n - 1)]
    yield rng.standard_normal(n)
    yield 1e200 * rng.standard_normal(n)
    yield 1e-200 * rng.standard_normal(n)
    yield np.r_[np.full(n // 3, 2.0), np.zeros(n // 3), -np.full(n - 2 * (n // 3), 0.5)]
    yield 10.0 ** rng.uniform(-16, 0, n) * rng.choice([-1.0, 1.0], n)


def _check(dims, project, seed, mu):
    rng = np.random.default_rng(seed)
    spectra = [list(_spectra(rng, d)) for d in dims]
    for k in range(len(spectra[0])):
        blocks = []
        for d, sp in zip(dims, spectra):
            q, _ = np.linalg.qr(rng.standard_normal((d, d)))
            m = (q * sp[k]) @ q.T
            blocks.append(0.5 * (m + m.T))
        x, z = project(np.concatenate([(m / mu).reshape(-1) for m in blocks]))
        o = 0
        for m in blocks:
            d = len(m)
            scale = np.abs(m).max() or 1.0
            w, v = np.linalg.eigh(m / scale)
            xb, zb = (mu * x[o:o + d * d].reshape(d, d) / scale, z[o:o + d * d].reshape(d, d) / scale)
            tol = 2e-14 * max(np.linalg.norm(m / scale), 1e-300)
            assert np.linalg.norm(xb - (v * np.maximum(w, 0)) @ v.T) <= tol, (d, k)
            assert np.linalg.norm(zb - (v * np.maximum(-w, 0)) @ v.T) <= tol, (d, k)
            assert np.linalg.eigvalsh(0.5 * (xb + xb.T))[0] >= -tol
            assert np.linalg.eigvalsh(0.5 * (zb + zb.T))[0] >= -tol
            o += d * d


@pytest.mark.parametrize("n,positivity", [(1, "D"), (2, "DQG"), (3, "DQG"), (5, "DQG"), (7, "DQ"), (8, "DQ")])
@pytest.mark.parametrize("mu", [1.0, 0.3])
def test_small_blocks_match_eigh(v2g, n, positivity, mu):
    import torch

    s = v2g.V2RDMSolver([n], (n + 1) // 2, (n + 1) // 2, options=dict(POSITIVITY=positivity))
    zero = torch.zeros(max(s.dimx, s.nconstraints), dtype=torch.float64, device="cuda")
    s.ATu(np.zeros(s.nconstraints))  # puts the tables on the device

    def project(x0):
        dx = torch.from_numpy(x0).cuda()
        dz = torch.full_like(dx, float("nan"))
        s.update_xz_noalloc(mu, zero.data_ptr(), zero.data_ptr(), dx.data_ptr(), dz.data_ptr())
        return dx.cpu().numpy(), dz.cpu().numpy()

    _check([d for d in s.dimensions if d > 0], project, 10 * n, mu)


@pytest.mark.parametrize("n,positivity", [(9, "DQ"), (7, "DQG"), (10, "DQG"), (13, "DQ"), (16, "D")])
def test_large_blocks_match_eigh(v2g, n, positivity):
    # blocks of 81, 98, 100 and 200, 169 and 78, 256 and 120: a team of CTAs each
    s = v2g.V2RDMSolver([n], (n + 1) // 2, (n + 1) // 2, options=dict(POSITIVITY=positivity))
    mu = 0.7

    def project(x0):
        s.set_state(x0, np.zeros(s.nconstraints), np.zeros(s.dimx), mu)
        s.update_xz(mu)
        x, _, z, _ = s.get_state()
        return x, z

    _check([d for d in s.dimensions if d > 0], project, n, mu)


def test_small_block_with_a_nan_is_nan(v2g):
    import torch

    s = v2g.V2RDMSolver([4], 2, 2)
    s.ATu(np.zeros(s.nconstraints))
    zero = torch.zeros(s.dimx, dtype=torch.float64, device="cuda")
    x0 = np.random.default_rng(0).standard_normal(s.dimx)
    x0[5] = np.nan  # in the first block
    dx = torch.from_numpy(x0).cuda()
    dz = torch.zeros_like(dx)
    s.update_xz_noalloc(1.0, zero.data_ptr(), zero.data_ptr(), dx.data_ptr(), dz.data_ptr())
    x, z = dx.cpu().numpy(), dz.cpu().numpy()
    first = int(s.dimensions[0]) ** 2
    assert np.isnan(x[:first]).any() and np.isnan(z[:first]).any()
    assert np.isfinite(x[first:]).all() and np.isfinite(z[first:]).all()

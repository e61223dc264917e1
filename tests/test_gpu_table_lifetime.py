"""A handle may go while a caller's stream still works on its constraint tables.

The batched maps and the allocation-free projection return at once.  Here many
of them are queued on a side stream, the handle is dropped (or given another
order of its orbitals, which rebuilds its tables), and other layouts are set up
and applied at once, so that memory given back too early would be handed out
again under the queued kernels.  Their results must be those of a handle that
stays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def others(v2g):
    """Other layouts' tables and workspaces, of the sizes that the dropped ones had."""
    for n in (12, 13, 14, 9, 11):
        s = v2g.V2RDMSolver([n], n // 2, n // 2)
        s.ATu(np.full(s.nconstraints, np.pi))


@pytest.mark.parametrize("how", ["drop", "reorder"])
def test_maps_after_their_handle(v2g, how):
    import torch

    n, nvec, length = 14, 12, 200

    def build():
        return v2g.V2RDMSolver([n], n // 2, n // 2)

    s = build()
    g = torch.Generator(device="cuda").manual_seed(5)
    u0 = torch.randn(s.dimx * nvec, dtype=torch.float64, device="cuda", generator=g)
    v0 = torch.randn(s.nconstraints * nvec, dtype=torch.float64, device="cuda", generator=g)
    outs = [torch.empty(k, dtype=torch.float64, device="cuda") for k in (v0.numel(), u0.numel())]
    side = torch.cuda.Stream()

    def queue(s, count):
        for _ in range(count):
            s.map_batched_device(nvec, u0.data_ptr(), outs[0].data_ptr(), side.cuda_stream)
            s.map_batched_device(nvec, v0.data_ptr(), outs[1].data_ptr(), side.cuda_stream, transpose=True)

    torch.cuda.synchronize()
    queue(s, 1)
    side.synchronize()
    want = [o.cpu().numpy() for o in outs]
    for o in outs:
        o.fill_(float("nan"))
    torch.cuda.synchronize()
    queue(s, length)
    if how == "drop":
        del s
    else:
        s.set_active_orbital_energies(np.arange(n, 0, -1, dtype=np.float64))
    others(v2g)
    side.synchronize()
    assert all(np.array_equal(w, o.cpu().numpy()) for w, o in zip(want, outs))


def test_projections_after_their_handle(v2g):
    import torch

    n, mu = 5, 1.3
    s = v2g.V2RDMSolver([n], n // 2, n // 2)
    rng = np.random.default_rng(6)
    y = rng.standard_normal(s.nconstraints)
    s.ATu(y)
    c, x0 = (torch.from_numpy(rng.standard_normal(s.dimx)).cuda() for _ in range(2))
    dy, x, z = torch.from_numpy(y).cuda(), torch.empty_like(c), torch.empty_like(c)
    side = torch.cuda.Stream()

    def queue(s, count):
        with torch.cuda.stream(side):
            for _ in range(count):
                x.copy_(x0)
                s.update_xz_noalloc(mu, c.data_ptr(), dy.data_ptr(), x.data_ptr(), z.data_ptr(), side.cuda_stream)

    torch.cuda.synchronize()
    queue(s, 1)
    side.synchronize()
    want = x.cpu().numpy(), z.cpu().numpy()
    queue(s, 300)
    del s
    others(v2g)
    side.synchronize()
    assert np.array_equal(want[0], x.cpu().numpy()) and np.array_equal(want[1], z.cpu().numpy())


@pytest.mark.parametrize("n", [4, 8, 12, 16])
def test_first_map_on_a_side_stream(v2g, n):
    """The tables are on the device before a caller's stream reads them: the
    first application of a layout is a handle's first call, on a stream that
    waits for no other."""
    import torch

    from helpers import csr_of

    s = v2g.V2RDMSolver([n], n // 2, n // 2, options=dict(CONSTRAIN_SPIN=n != 12))
    A = csr_of(s)
    y = np.random.default_rng(n).standard_normal(s.nconstraints)
    d_in, d_out = torch.from_numpy(y).cuda(), torch.empty(s.dimx, dtype=torch.float64, device="cuda")
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    s.map_batched_device(1, d_in.data_ptr(), d_out.data_ptr(), side.cuda_stream, transpose=True)
    side.synchronize()
    want = A.T @ y
    assert np.abs(d_out.cpu().numpy() - want).max() <= 1e-12 * np.abs(want).max()
